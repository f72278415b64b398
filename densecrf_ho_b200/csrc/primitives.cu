// Deterministic device-wide integer primitives (no float atomics anywhere).
#include <algorithm>

#include "primitives.cuh"

namespace dcrf {

namespace {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;
constexpr unsigned kFull = 0xffffffffu;

// Exclusive scan of one int per thread across a 256-thread block; also
// returns the block total.
__device__ __forceinline__ int block_exclusive_scan(int v, int* warp_tot, int* total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(kFull, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_tot[w] = x;
    __syncthreads();
    if (w == 0) {
        int s = lane < kScanThreads / 32 ? warp_tot[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int y = __shfl_up_sync(kFull, s, o);
            if (lane >= o) s += y;
        }
        if (lane < kScanThreads / 32) warp_tot[lane] = s;
    }
    __syncthreads();
    int prefix = w ? warp_tot[w - 1] : 0;
    *total = warp_tot[kScanThreads / 32 - 1];
    return prefix + x - v;
}

__global__ void scan_reduce_kernel(const int* __restrict__ in, int n, int* __restrict__ bsum) {
    __shared__ int wt[kScanThreads / 32];
    long base = (long)blockIdx.x * kScanTile;
    int s = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
        long idx = base + (long)threadIdx.x * kScanItems + i;
        if (idx < n) s += in[idx];
    }
    int tot;
    block_exclusive_scan(s, wt, &tot);
    if (threadIdx.x == 0) bsum[blockIdx.x] = tot;
}

// Single block: in-place exclusive scan of the per-tile sums.
__global__ void scan_top_kernel(int* __restrict__ bsum, int nb, int* __restrict__ d_total) {
    __shared__ int wt[kScanThreads / 32];
    int carry = 0;
    for (int base = 0; base < nb; base += kScanTile) {
        int v[kScanItems];
        int s = 0;
#pragma unroll
        for (int i = 0; i < kScanItems; i++) {
            int idx = base + threadIdx.x * kScanItems + i;
            v[i] = idx < nb ? bsum[idx] : 0;
            s += v[i];
        }
        int tot;
        int ex = block_exclusive_scan(s, wt, &tot);
        int run = carry + ex;
#pragma unroll
        for (int i = 0; i < kScanItems; i++) {
            int idx = base + threadIdx.x * kScanItems + i;
            if (idx < nb) bsum[idx] = run;
            run += v[i];
        }
        carry += tot;
        __syncthreads();
    }
    if (threadIdx.x == 0 && d_total) *d_total = carry;
}

// A thread's items are neighbours: 16 bytes at a time where the arrays allow
// (vec): 11.6 -> 5.9 us for 1.84 M.
__global__ void scan_apply_kernel(const int* in, int* out, int n, const int* __restrict__ bsum, int vec) {
    static_assert(kScanItems % 4 == 0, "whole 16-byte accesses per thread");
    __shared__ int wt[kScanThreads / 32];
    const long base = (long)blockIdx.x * kScanTile + (long)threadIdx.x * kScanItems;
    const bool whole = vec && base + kScanItems <= n;
    int v[kScanItems];
    int s = 0;
    if (whole) {
#pragma unroll
        for (int i = 0; i < kScanItems; i += 4) {
            const int4 x = *reinterpret_cast<const int4*>(in + base + i);
            v[i] = x.x;
            v[i + 1] = x.y;
            v[i + 2] = x.z;
            v[i + 3] = x.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < kScanItems; i++) v[i] = base + i < n ? in[base + i] : 0;
    }
#pragma unroll
    for (int i = 0; i < kScanItems; i++) s += v[i];
    int tot;
    int run = bsum[blockIdx.x] + block_exclusive_scan(s, wt, &tot);
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
        const int c = v[i];
        v[i] = run;
        run += c;
    }
    if (whole) {
#pragma unroll
        for (int i = 0; i < kScanItems; i += 4)
            *reinterpret_cast<int4*>(out + base + i) = make_int4(v[i], v[i + 1], v[i + 2], v[i + 3]);
    } else {
#pragma unroll
        for (int i = 0; i < kScanItems; i++)
            if (base + i < n) out[base + i] = v[i];
    }
}

static int int4_ok(const int* a, const int* b) {
    return (reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) % 16 == 0;
}

// ---------------------------------------------------------------- sort --
constexpr int kSortThreads = 256;
constexpr int kSortItems = 8;
constexpr int kSortTile = kSortThreads * kSortItems;
constexpr int kRadix = 256;

// Histogram of one digit per tile; all of a thread's keys are loaded before
// they are counted.
__global__ void __launch_bounds__(kSortThreads)
    radix_hist_kernel(const int* __restrict__ keys, int n, int shift, int ntiles, int* __restrict__ hist) {
    __shared__ int h[kRadix];
    for (int i = threadIdx.x; i < kRadix; i += blockDim.x) h[i] = 0;
    __syncthreads();
    const long base = (long)blockIdx.x * kSortTile;
    int k[kSortItems];
#pragma unroll
    for (int i = 0; i < kSortItems; i++) {
        const long idx = base + i * kSortThreads + threadIdx.x;
        k[i] = idx < n ? (keys[idx] >> shift) & (kRadix - 1) : -1;
    }
#pragma unroll
    for (int i = 0; i < kSortItems; i++)
        if (k[i] >= 0) atomicAdd(&h[k[i]], 1);
    __syncthreads();
    for (int i = threadIdx.x; i < kRadix; i += blockDim.x) hist[(long)i * ntiles + blockIdx.x] = h[i];
}

// One block per digit: exclusive scan of the digit's tile counts in place, its
// total to hist[kRadix * ntiles + digit].  The scatter adds the totals of the
// smaller digits, so the scan needs one launch.
__global__ void __launch_bounds__(kScanThreads) radix_row_scan_kernel(int* __restrict__ hist, int ntiles) {
    __shared__ int wt[kScanThreads / 32];
    int* row = hist + (long)blockIdx.x * ntiles;
    int carry = 0;
    for (int base = 0; base < ntiles; base += kScanThreads) {
        const int i = base + threadIdx.x;
        const int v = i < ntiles ? row[i] : 0;
        int tot;
        const int ex = block_exclusive_scan(v, wt, &tot);
        if (i < ntiles) row[i] = carry + ex;
        carry += tot;
        __syncthreads();  // wt is rewritten
    }
    if (threadIdx.x == 0) hist[(long)kRadix * ntiles + blockIdx.x] = carry;
}

// Stable scatter.  Each warp ranks 512 consecutive elements of the tile among
// equal digits in index order (warp match + its own counts, no block barrier),
// then the warps' counts are scanned per digit and the tile is put in digit
// order in shared memory, from where a warp writes runs of neighbours (single
// four-byte stores all over the output were 32 passes through L1 a warp each).
// Latency-bound: two blocks of 4096 elements at 103 registers left 450 tiles
// in one and a half waves.  With 2048 elements, six blocks fit and a 640x480
// bilateral lattice's 1.84 M entries take one wave: 26.3 -> 22.5 us by the
// staging, -> 13.7 by the size; 320x240 13.8 -> 7.3 us.  vals_in null: the
// value is the index.
__global__ void __launch_bounds__(kSortThreads, 6)
    radix_scatter_kernel(const int* __restrict__ keys_in, const int* __restrict__ vals_in, int n, int shift,
                         int ntiles, const int* __restrict__ offs, int* __restrict__ keys_out,
                         int* __restrict__ vals_out) {
    constexpr int W = kSortThreads / 32;
    __shared__ int cnt[W][kRadix];
    __shared__ int to_out[kRadix];
    __shared__ int sk[kSortTile], sv[kSortTile];
    __shared__ int wt[kScanThreads / 32];
    static_assert(kSortThreads == kRadix && kScanThreads == kSortThreads, "thread d owns digit d");
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, t = threadIdx.x;
#pragma unroll
    for (int i = 0; i < W; i++) cnt[i][t] = 0;
    const long base = (long)blockIdx.x * kSortTile + (long)w * (kSortTile / W);
    int key[kSortItems], rank[kSortItems];
#pragma unroll
    for (int i = 0; i < kSortItems; i++) {
        const long idx = base + i * 32 + lane;
        key[i] = idx < n ? keys_in[idx] : 0;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kSortItems; i++) {
        const bool valid = base + i * 32 + lane < n;
        const int dig = valid ? (key[i] >> shift) & (kRadix - 1) : kRadix;
        const unsigned peers = __match_any_sync(kFull, dig);
        rank[i] = __popc(peers & ((1u << lane) - 1u)) + (valid ? cnt[w][dig] : 0);
        __syncwarp();
        if (valid && (__ffs(peers) - 1) == lane) cnt[w][dig] += __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    {  // thread t: digit t's bases over the digits and warps before it, in the tile and overall
        int tot, count = 0;
#pragma unroll
        for (int i = 0; i < W; i++) count += cnt[i][t];
        int run = block_exclusive_scan(count, wt, &tot);
        const int local = run;
#pragma unroll
        for (int i = 0; i < W; i++) {
            const int c = cnt[i][t];
            cnt[i][t] = run;
            run += c;
        }
        __syncthreads();  // wt is rewritten
        const int total = offs[(long)kRadix * ntiles + t];
        to_out[t] = block_exclusive_scan(total, wt, &tot) + offs[(long)t * ntiles + blockIdx.x] - local;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kSortItems; i++) {
        const long idx = base + i * 32 + lane;
        if (idx < n) {
            const int o = cnt[w][(key[i] >> shift) & (kRadix - 1)] + rank[i];
            sk[o] = key[i];
            sv[o] = vals_in ? vals_in[idx] : (int)idx;
        }
    }
    __syncthreads();
    const int here = (int)min((long)kSortTile, n - (long)blockIdx.x * kSortTile);
#pragma unroll
    for (int i = 0; i < kSortItems; i++) {
        const int p = i * kSortThreads + t;
        if (p < here) {
            const int k = sk[p];
            const int o = to_out[(k >> shift) & (kRadix - 1)] + p;
            keys_out[o] = k;
            vals_out[o] = sv[p];
        }
    }
}

// First flags (lattice.cu): flag[e] = [table[slot[e]] == e] and their sums per
// scan tile, in one pass.
__global__ void flag_reduce_kernel(const int* __restrict__ slot, const int* __restrict__ table, int n,
                                   int* __restrict__ flag, int* __restrict__ bsum) {
    __shared__ int wt[kScanThreads / 32];
    const long base = (long)blockIdx.x * kScanTile;
    int s = 0, f[kScanItems];
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
        const long e = base + i * kScanThreads + threadIdx.x;
        f[i] = e < n ? slot[e] : -1;
    }
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
        const long e = base + i * kScanThreads + threadIdx.x;
        f[i] = f[i] >= 0 && table[f[i]] == (int)e;
        s += f[i];
        if (e < n) flag[e] = f[i];
    }
    int tot;
    block_exclusive_scan(s, wt, &tot);
    if (threadIdx.x == 0) bsum[blockIdx.x] = tot;
}

}  // namespace

void exclusive_scan(const int* in, int* out, int n, int* d_total, ScanScratch& s, cudaStream_t st) {
    if (n <= 0) {
        if (d_total) DCRF_CUDA(cudaMemsetAsync(d_total, 0, sizeof(int), st));
        return;
    }
    int nb = ceil_div(n, kScanTile);
    int* bs = s.block_sums.ensure(nb);
    launch(scan_reduce_kernel, nb, kScanThreads, 0, st, in, n, bs);
    launch(scan_top_kernel, 1, kScanThreads, 0, st, bs, nb, d_total);
    launch(scan_apply_kernel, nb, kScanThreads, 0, st, in, out, n, (const int*)bs, int4_ok(in, out));
    DCRF_LAUNCH_CHECK();
}

void first_flags_scan(const int* slot, const int* table, int n, int* ranks, int* d_total, ScanScratch& s,
                      cudaStream_t st) {
    const int nb = ceil_div(n, kScanTile);
    int* bs = s.block_sums.ensure(nb);
    launch(flag_reduce_kernel, nb, kScanThreads, 0, st, slot, table, n, ranks, bs);
    launch(scan_top_kernel, 1, kScanThreads, 0, st, bs, nb, d_total);
    launch(scan_apply_kernel, nb, kScanThreads, 0, st, (const int*)ranks, ranks, n, (const int*)bs,
           int4_ok(ranks, ranks));
    DCRF_LAUNCH_CHECK();
}

// Sorts (kin, vin) -- vin null: the indexes -- by passes that write alternately
// to `a` and `b` buffers; returns true when the result is in a.
static bool radix_passes(const int* kin, const int* vin, int* ka, int* va, int* kb, int* vb, int n, int key_bits,
                         SortScratch& s, cudaStream_t st) {
    const int ntiles = ceil_div(n, kSortTile);
    int* hist = s.hist.ensure((size_t)kRadix * (ntiles + 1));
    bool to_a = true;
    for (int shift = 0; shift < key_bits; shift += 8) {
        int *ko = to_a ? ka : kb, *vo = to_a ? va : vb;
        launch(radix_hist_kernel, ntiles, kSortThreads, 0, st, kin, n, shift, ntiles, hist);
        launch(radix_row_scan_kernel, kRadix, kScanThreads, 0, st, hist, ntiles);
        launch(radix_scatter_kernel, ntiles, kSortThreads, 0, st, kin, vin, n, shift, ntiles, (const int*)hist, ko,
               vo);
        kin = ko;
        vin = vo;
        to_a = !to_a;
    }
    DCRF_LAUNCH_CHECK();
    return !to_a;
}

void radix_sort_pairs(int* keys, int* vals, int n, int key_bits, SortScratch& s, cudaStream_t st) {
    if (n <= 1 || key_bits <= 0) return;
    int* ka = s.keys_alt.ensure(n);
    int* va = s.vals_alt.ensure(n);
    if (radix_passes(keys, vals, ka, va, keys, vals, n, key_bits, s, st)) {
        DCRF_CUDA(cudaMemcpyAsync(keys, ka, sizeof(int) * n, cudaMemcpyDeviceToDevice, st));
        DCRF_CUDA(cudaMemcpyAsync(vals, va, sizeof(int) * n, cudaMemcpyDeviceToDevice, st));
    }
}

void radix_sort_index(const int* keys, int n, int key_bits, int* kbuf, int* vbuf, const int** keys_out,
                      const int** vals_out, SortScratch& s, cudaStream_t st) {
    int* ka = s.keys_alt.ensure(std::max(n, 1));
    int* va = s.vals_alt.ensure(std::max(n, 1));
    const bool in_a = radix_passes(keys, nullptr, ka, va, kbuf, vbuf, n, std::max(key_bits, 1), s, st);
    *keys_out = in_a ? ka : kbuf;
    *vals_out = in_a ? va : vbuf;
}

}  // namespace dcrf
