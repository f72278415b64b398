// Permutohedral lattice construction and filtering on sm_100a.
//
// Construction reproduces Permutohedral::init's SSE path
// (src/permutohedral.cpp:152-333) bit for bit:
//   K1 elevate   one thread per pixel: elevation, rounding to the nearest
//                0-coloured vertex (round-to-nearest-even, as _mm_cvtps_epi32
//                does), rank, barycentric weights and the d+1 vertex keys;
//                the pixel count is padded to a multiple of 4 with zero
//                features, like the reference's last SSE block.
//   K2 insert    open-addressing hash insert of every (pixel, remainder)
//                entry; each slot ends up holding the SMALLEST entry index
//                with its key (atomicMin), i.e. the key's first occurrence.
//   K3 compact   vertex id = rank of the first occurrence among all first
//                occurrences (flag + exclusive scan) -- exactly the
//                insertion order HashTable::find produces (:100-128).
//   K4 neighbours  per (axis, vertex) lookup of key -1/+d and key +1/-d
//                (:316-330).
//   K5 splat lists  stable radix sort of entries by vertex id.
// Filtering reproduces sseCompute (L > 2) / seqCompute (L <= 2)
// (src/permutohedral.cpp:998-1058 / 488-540) and the 10-bin ordered filter
// (:548-701) with the same per-element operation order, so results are
// identical to the reference, with no float atomics.
#include <algorithm>
#include <cmath>
#include <mutex>
#include <string>
#include <vector>

#include "lattice.cuh"

namespace dcrf {

namespace {

constexpr int kEmpty = -1;
constexpr int kRes = 10;       // RESOLUTION (include/permutohedral.h:41)
constexpr int kOrdW = 2 * kRes;  // lower + upper bins per (vertex, label)
constexpr int kStageWarps = 2;   // warps (splat lists) per splat block
constexpr int kStages = 3;       // shared-memory ring depth, in chunks
constexpr int kChunk = 32;       // entries per chunk (13 KB of ring per warp: 16 warps / SM)
constexpr int kMaxOrderKey = (1 << 24) - 1;
constexpr int kLongList = 64;    // lists longer than this use the staged warp kernels
constexpr int kHugeList = 1024;  // lists longer than this get a block (plain) or the finest split (ordered splat)
constexpr int kHugeLabels = 12;  // labels per block for those lists (120 threads)
constexpr int kTB = 256;         // threads per block of the element-wise kernels
constexpr int kSegPad = 4;       // entries past the splat lists' end that a paired load may touch

template <int KW>
struct Key {
    int4 w[KW];
};

template <int KW>
__device__ __forceinline__ Key<KW> load_key(const int4* __restrict__ k, long e) {
    Key<KW> r;
#pragma unroll
    for (int i = 0; i < KW; i++) r.w[i] = __ldg(k + e * KW + i);
    return r;
}

template <int KW>
__device__ __forceinline__ bool key_eq(const Key<KW>& a, const Key<KW>& b) {
    bool eq = true;
#pragma unroll
    for (int i = 0; i < KW; i++)
        eq &= (a.w[i].x == b.w[i].x) & (a.w[i].y == b.w[i].y) & (a.w[i].z == b.w[i].z) &
              (a.w[i].w == b.w[i].w);
    return eq;
}

__device__ __forceinline__ uint32_t mix32(uint32_t h) {
    h ^= h >> 16;
    h *= 0x85ebca6bu;
    h ^= h >> 13;
    h *= 0xc2b2ae35u;
    h ^= h >> 16;
    return h;
}

template <int KW>
__device__ __forceinline__ uint32_t key_hash(const Key<KW>& k) {
    uint32_t h = 0x9e3779b9u;
#pragma unroll
    for (int i = 0; i < KW; i++) {
        h = mix32(h ^ (uint32_t)k.w[i].x);
        h = mix32(h ^ (uint32_t)k.w[i].y);
        h = mix32(h ^ (uint32_t)k.w[i].z);
        h = mix32(h ^ (uint32_t)k.w[i].w);
    }
    return h;
}

template <int KW>
__device__ __forceinline__ void key_set(Key<KW>& k, int c, int16_t v) {
    int* words = reinterpret_cast<int*>(k.w);
    int wi = c >> 1;
    uint32_t u = (uint32_t)words[wi];
    if (c & 1) u = (u & 0x0000ffffu) | ((uint32_t)(uint16_t)v << 16);
    else u = (u & 0xffff0000u) | (uint32_t)(uint16_t)v;
    words[wi] = (int)u;
}

template <int KW>
__device__ __forceinline__ int16_t key_get(const Key<KW>& k, int c) {
    const int* words = reinterpret_cast<const int*>(k.w);
    uint32_t u = (uint32_t)words[c >> 1];
    return (int16_t)(uint16_t)((c & 1) ? (u >> 16) : (u & 0xffffu));
}

template <int KW>
__device__ __forceinline__ void key_zero(Key<KW>& k) {
#pragma unroll
    for (int i = 0; i < KW; i++) k.w[i] = make_int4(0, 0, 0, 0);
}

// _mm_cvtps_epi32 (round to nearest even; out-of-range -> INT_MIN) and back.
__device__ __forceinline__ float cvt_rne(float v) {
    if (!(fabsf(v) < 2147483648.0f)) return -2147483648.0f;
    return (float)__float2int_rn(v);
}

// K1: one thread per (padded) pixel.
template <int DM>
__global__ void elevate_kernel(const float* __restrict__ feat, int N, int Np, int d,
                               const float* __restrict__ scale, int4* __restrict__ ekeys,
                               int* __restrict__ rank_out, float* __restrict__ bary_out) {
    constexpr int KW = (DM + 7) / 8;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= Np) return;
    const int d1 = d + 1;
    const float invdp1 = 1.0f / (float)d1, dp1 = (float)d1;
    float f[DM], el[DM + 1], rem0[DM + 1], rk[DM + 1], b[DM + 2];
    for (int j = 0; j < d; j++) f[j] = k < N ? feat[(long)k * d + j] : 0.0f;
    // Elevation (:213-219): sm accumulates from the last coordinate down.
    float sm = 0.0f;
    for (int j = d; j > 0; j--) {
        float cf = fmul(f[j - 1], scale[j - 1]);
        el[j] = fsub(sm, fmul((float)j, cf));
        sm = fadd(sm, cf);
    }
    el[0] = sm;
    // Closest 0-coloured simplex (:222-232).
    float sum = 0.0f;
    for (int i = 0; i <= d; i++) {
        float v = cvt_rne(fmul(invdp1, el[i]));
        rem0[i] = fmul(v, dp1);
        sum = fadd(sum, v);
    }
    // Rank (:235-245).
    for (int i = 0; i <= d; i++) rk[i] = 0.0f;
    for (int i = 0; i < d; i++) {
        float di = fsub(el[i], rem0[i]);
        for (int j = i + 1; j <= d; j++) {
            float dj = fsub(el[j], rem0[j]);
            float c = (di < dj) ? 1.0f : 0.0f;
            rk[i] = fadd(rk[i], c);
            rk[j] = fadd(rk[j], fsub(1.0f, c));
        }
    }
    // Back onto the plane (:248-254).
    for (int i = 0; i <= d; i++) {
        rk[i] = fadd(rk[i], sum);
        float add = rk[i] < 0.0f ? dp1 : 0.0f;
        float sub = rk[i] >= dp1 ? dp1 : 0.0f;
        float t = fsub(add, sub);
        rk[i] = fadd(rk[i], t);
        rem0[i] = fadd(rem0[i], t);
    }
    // Barycentric coordinates (:257-275).
    for (int i = 0; i < d + 2; i++) b[i] = 0.0f;
    for (int i = 0; i <= d; i++) {
        float v = fmul(fsub(el[i], rem0[i]), invdp1);
        int p = (int)fsub((float)d, rk[i]);
        p = min(max(p, 0), d);  // in range for finite features; guards NaN input
        b[p] = fadd(b[p], v);
        b[p + 1] = fsub(b[p + 1], v);
    }
    b[0] = fadd(b[0], fadd(1.0f, b[d + 1]));
    // Keys of the d+1 vertices (:280-287); canonical simplex (:183-188).
    for (int r = 0; r <= d; r++) {
        Key<KW> key;
        key_zero(key);
        for (int i = 0; i < d; i++) {
            int ri = (int)rk[i];
            int canon = (ri <= d - r) ? r : r - d1;
            key_set(key, i, (int16_t)(int)fadd(rem0[i], (float)canon));
        }
        long e = (long)k * d1 + r;
#pragma unroll
        for (int w = 0; w < KW; w++) ekeys[e * KW + w] = key.w[w];
        if (k < N) {
            rank_out[e] = (int)rk[r];
            bary_out[e] = b[r];
        }
    }
}

// K2: insert every entry; slots keep the smallest entry index of their key.
template <int KW>
__global__ void insert_kernel(const int4* __restrict__ ekeys, int E, int* table, unsigned mask,
                              int* __restrict__ entry_slot) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= E) return;
    const Key<KW> key = load_key<KW>(ekeys, e);
    unsigned h = key_hash(key) & mask;
    for (unsigned probe = 0; probe <= mask; probe++) {  // bounded: table is never full
        int cur = *(volatile int*)(table + h);
        if (cur == kEmpty) {
            int old = atomicCAS(table + h, kEmpty, e);
            if (old == kEmpty) {
                entry_slot[e] = (int)h;
                return;
            }
            cur = old;
        }
        if (key_eq(load_key<KW>(ekeys, cur), key)) {
            atomicMin(table + h, e);
            entry_slot[e] = (int)h;
            return;
        }
        h = (h + 1) & mask;
    }
}

__global__ void first_flag_kernel(int E, const int* __restrict__ entry_slot,
                                  const int* __restrict__ table, int* __restrict__ flag) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= E) return;
    flag[e] = table[entry_slot[e]] == e ? 1 : 0;
}

// K3: vertex ids and vertex keys.
template <int KW>
__global__ void finalize_kernel(int E, int Ereal, int d, const int* __restrict__ entry_slot,
                                const int* __restrict__ table, const int* __restrict__ first_rank,
                                const int4* __restrict__ ekeys, int* __restrict__ offset,
                                int16_t* __restrict__ vkeys, int* __restrict__ slot_vid) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= E) return;
    const int s = entry_slot[e];
    const int f = table[s];
    const int vid = first_rank[f];
    if (e < Ereal) offset[e] = vid;
    if (f == e) {
        slot_vid[s] = vid;
        const Key<KW> key = load_key<KW>(ekeys, e);
        for (int c = 0; c < d; c++) vkeys[(long)vid * d + c] = key_get(key, c);
    }
}

template <int KW>
__device__ __forceinline__ int lookup(const Key<KW>& key, const int* __restrict__ table,
                                      unsigned mask, const int4* __restrict__ ekeys,
                                      const int* __restrict__ slot_vid) {
    unsigned h = key_hash(key) & mask;
    for (unsigned probe = 0; probe <= mask; probe++) {
        int cur = table[h];
        if (cur == kEmpty) return -1;
        if (key_eq(load_key<KW>(ekeys, cur), key)) return slot_vid[h];
        h = (h + 1) & mask;
    }
    return -1;
}

// K4: blur neighbours, stored shifted by one (0 = absent).
template <int KW>
__global__ void neighbor_kernel(int M, int d, const int16_t* __restrict__ vkeys,
                                const int* __restrict__ table, unsigned mask,
                                const int4* __restrict__ ekeys, const int* __restrict__ slot_vid,
                                int2* __restrict__ nbr) {
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long)(d + 1) * M) return;
    const int j = (int)(t / M), v = (int)(t - (long)j * M);
    Key<KW> n1, n2;
    key_zero(n1);
    key_zero(n2);
    for (int c = 0; c < d; c++) {
        int kc = vkeys[(long)v * d + c];
        int a = c == j ? kc + d : kc - 1;
        int bb = c == j ? kc - d : kc + 1;
        key_set(n1, c, (int16_t)a);
        key_set(n2, c, (int16_t)bb);
    }
    int i1 = lookup(n1, table, mask, ekeys, slot_vid);
    int i2 = lookup(n2, table, mask, ekeys, slot_vid);
    nbr[t] = make_int2(i1 + 1, i2 + 1);
}

__global__ void count_kernel(int E, const int* __restrict__ offset, int* __restrict__ counts) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e < E) atomicAdd(counts + offset[e], 1);
}

__global__ void iota_copy_kernel(int E, const int* __restrict__ offset, int* __restrict__ keys,
                                 int* __restrict__ vals) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= E) return;
    keys[e] = offset[e];
    vals[e] = e;
}

// A splat list's entry is (pixel, weight bits).
__device__ __forceinline__ float entry_w(int2 e) { return __int_as_float(e.y); }

__global__ void seg_fill_kernel(int E, int d1, const int* __restrict__ sorted_entries,
                                const float* __restrict__ bary, int2* __restrict__ seg) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= E) return;
    const int e = sorted_entries[s];
    seg[s] = make_int2(e / d1, __float_as_int(bary[e]));
}

// ------------------------------------------------------------- filter --

// Splat as a gather: value(v, k) = sum over v's entries, in entry order, of
// w * in[p][k] (times the symmetric normalisation when pre_norm is given,
// which DenseKernel::filter applies before the lattice, src/pairwise.cpp:61).
//
// One warp per vertex, lanes = labels (in chunks of 32).  The sum must stay
// sequential in entry order to reproduce the reference's scatter, so each
// lane's float adds form one dependent chain; everything else is kept off
// that chain.  The list is streamed in chunks of 32 entries through a ring
// of kStages shared-memory buffers with cp.async: while chunk c is summed,
// chunks c+1 .. c+kStages-1 (up to 96 entries x L values, plus their weights
// and normalisation factors) are in flight, so a single long list is not
// serialised on L2 latency.  Vertices are visited longest list first
// (`order`) so the few very long lists of a coarse lattice start early.
// The filter kernels loop over their units (list positions, vertices,
// pixels or tiles) with a grid-stride loop: one pass with a full grid, or,
// in a batched solve, the units of the images still running (Live) with a
// grid sized for the device.

__device__ __forceinline__ unsigned smem_addr(const void* p) {
    return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void cp_async4(void* sdst, const void* gsrc) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(smem_addr(sdst)), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async8(void* sdst, const void* gsrc) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(smem_addr(sdst)), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// Streams the list [s0, s1) of one vertex through the per-warp ring:
// `vals_of(slot, e)` is this lane's staged word for entry e, and
// consume(slot, n) is called once per chunk, in order.
template <typename T, typename Consume>
__device__ __forceinline__ void stream_list(int s0, int s1, int L, int k, bool act, int lane,
                                            const int2* __restrict__ seg,
                                            const T* __restrict__ src, T (*ring)[kChunk][32], float (*mw)[kChunk],
                                            Consume&& consume) {
    const int nch = (s1 - s0 + kChunk - 1) / kChunk;
    auto pix_of = [&](int c) {
        const int base = s0 + c * kChunk;
        return (c < nch && lane < s1 - base) ? seg[base + lane].x : 0;
    };
    auto issue = [&](int c, int pc) {
        const int slot = c % kStages, base = s0 + c * kChunk, n = min(kChunk, s1 - base);
        if (lane < n) cp_async4(&mw[slot][lane], &seg[base + lane].y);
        for (int e = 0; e < n; e++) {
            const int p = __shfl_sync(0xffffffffu, pc, e);
            if (act) cp_async4(&ring[slot][e][lane], src + (long)p * L + k);
        }
    };
    int pcur = pix_of(0);
#pragma unroll
    for (int c = 0; c < kStages - 1; c++) {
        const int pn = pix_of(c + 1);
        if (c < nch) issue(c, pcur);
        cp_async_commit();
        pcur = pn;
    }
    for (int c = 0; c < nch; c++) {
        const int ci = c + kStages - 1;
        const int pn = pix_of(ci + 1);
        if (ci < nch) issue(ci, pcur);
        cp_async_commit();
        pcur = pn;
        cp_async_wait<kStages - 1>();  // chunk c has landed (this lane's copies)
        __syncwarp();                  // ... and every other lane's
        consume(c % kStages, min(kChunk, s1 - (s0 + c * kChunk)));
        __syncwarp();                  // the slot is refilled kStages-1 chunks later
    }
    cp_async_wait<0>();
    __syncwarp();
}

// The allocation-free filter's splat of the long lists (it may not hold the
// padded rows of the splat below): rows as they are, one warp per vertex.
__global__ void __launch_bounds__(32 * kStageWarps)
    splat_kernel(int M, int L, const int* __restrict__ order, const int* __restrict__ seg_start,
                 const int2* __restrict__ seg, const float* __restrict__ in,
                 float* __restrict__ vals) {
    __shared__ float ring[kStageWarps][kStages][kChunk][32];
    __shared__ float mw[kStageWarps][kStages][kChunk];
    const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int unit = blockIdx.x * kStageWarps + wib;
    if (unit >= M) return;  // warp-uniform
    const int v = order[unit];
    const int s0 = seg_start[v], s1 = seg_start[v + 1];
    for (int kb = 0; kb < L; kb += 32) {
        const int k = kb + lane;
        const bool act = k < L;
        float acc = 0.0f;
        stream_list<float>(s0, s1, L, k, act, lane, seg, in, ring[wib], mw[wib], [&](int slot, int n) {
#pragma unroll 4
            for (int e = 0; e < n; e++) acc = fadd(acc, fmul(mw[wib][slot][e], ring[wib][slot][e][lane]));
        });
        if (act) vals[(long)(v + 1) * L + k] = acc;
    }
}

// ... and of the short lists: one thread per (vertex, label).
__global__ void splat_short_kernel(int n_short, int L, const int* __restrict__ order,
                                   const int* __restrict__ seg_start, const int2* __restrict__ seg, const float* __restrict__ in,
                                   float* __restrict__ vals) {
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long)n_short * L) return;
    const int u = (int)(t / L), k = (int)(t - (long)u * L);
    const int v = order[u];
    const int s0 = seg_start[v], s1 = seg_start[v + 1];
    float acc = 0.0f;
#pragma unroll 4
    for (int s = s0; s < s1; s++) acc = fadd(acc, fmul(entry_w(seg[s]), in[(long)seg[s].x * L + k]));
    vals[(long)(v + 1) * L + k] = acc;
}

// ----------------------------------------------------------- row splat --
// The plain splat, L > 2.  The input is copied once into rows of Q = ceil(L /
// 4) float4 (pad_rows_kernel: labels past L are zero, the normalisation
// factor already applied: fmul(x, norm) is the product the reference forms
// before the splat), so that a list entry costs Q aligned 16-byte loads
// instead of L scalar ones plus a norm gather.  L = 21, one warp instruction
// per entry and label group:
//   short lists  one thread per (vertex, four labels), kSplatU entries' rows
//                in flight, the next entries' (pixel, weight) already loaded;
//   long lists   one warp per vertex, a ring of kSplatStages chunks of 32
//                entries filled with 16-byte cp.async (6 per lane and chunk
//                for L = 21), lane = label for the sums: 1 shared-memory read
//                + 1 multiply + 1 add per entry;
//   huge lists   one block per vertex: the block's whole ring for one list
//                (kHugeStages chunks of 64 entries), four warps copying and the
//                first one adding.  A lone warp with two chunks of lookahead
//                waits for its loads (about 840 cycles per 32 entries: the
//                3607-entry list of a 640x480 bilateral lattice set the
//                splat's 50 us); with five chunks of 64 in flight the chain of
//                dependent adds is what is left.
// All sum a (vertex, label)'s entries in list order from +0, one rounding per
// product and per sum, as the reference's scatter does.
constexpr int kSplatU = 4;        // entries in flight per thread (short lists)
constexpr int kSplatWarps = 4;    // lists per block (long lists)
constexpr int kSplatStages = 3;   // 9.4 KB of ring per warp at L = 21: 20 warps / SM
constexpr int kSplatThreads = 32 * kSplatWarps;

__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
// a + w x per half, the product and the sum each rounded: scalar products and
// a packed sum.  A packed product feeding a packed sum was measured to come
// out as one fused multiply-add (rounded once), which the reference's SSE2
// arithmetic does not do.
__device__ __forceinline__ unsigned long long add_mul2(unsigned long long a, float w, unsigned long long x) {
    const float2 f = unpack2(x);
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(pack2(fmul(w, f.x), fmul(w, f.y))));
    return r;
}

__device__ __forceinline__ void cp_async16(void* sdst, const void* gsrc) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem_addr(sdst)), "l"(gsrc) : "memory");
}

// A batched solve's live slice tiles, or tiles of the whole pixel range: the
// first pixel of tile u and its pixel count.
__device__ __forceinline__ int tile_pixels(const Live& lv, const long* pix_base, long u, int tile, long N,
                                           long& p0) {
    long pend = N;
    if (lv.n) {
        long local;
        const int img = live_locate(lv, u, local);
        p0 = pix_base[img] + local * tile;
        pend = pix_base[img + 1];
    } else {
        p0 = u * tile;
    }
    return (int)min((long)tile, pend - p0);
}

// rows[i][q] = (in[i][4q .. 4q+3] o norm[i]), zero past L: a tile of pixels per
// warp, copied to shared memory as it lies (16 bytes at a time where the
// pointer allows, vec) and written back in rows.  Bound by memory: 84 bytes
// in, 96 out per pixel at L = 21.
constexpr int kPadWarps = 4;
template <int QC>
__global__ void __launch_bounds__(32 * kPadWarps)
    pad_rows_kernel(int N, int L, int Qrt, int tile, const float* __restrict__ in, const float* __restrict__ norm,
                    float4* __restrict__ rows, Live lv, const long* __restrict__ pix_base, int vec) {
    extern __shared__ __align__(16) unsigned char pad_smem[];
    const int Q = QC ? QC : Qrt;
    const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float* buf = reinterpret_cast<float*>(pad_smem) + (size_t)wib * ((tile * L + 3) & ~3);
    grid_release();
    grid_wait();
    const long total = live_total(lv, ((long)N + tile - 1) / tile);
    for (long u = (long)blockIdx.x * kPadWarps + wib; u < total; u += (long)gridDim.x * kPadWarps) {
        long p0;
        const int np = tile_pixels(lv, pix_base, u, tile, N, p0);
        const long t0 = p0 * L;
        const int ne = np * L, n4 = vec && (t0 & 3) == 0 ? ne >> 2 : 0;
        for (int e = lane; e < n4; e += 32) cp_async16(buf + 4 * e, in + t0 + 4 * e);
        for (int e = 4 * n4 + lane; e < ne; e += 32) cp_async4(buf + e, in + t0 + e);
        cp_async_commit();
        cp_async_wait<0>();
        __syncwarp();
        for (int it = lane; it < np * Q; it += 32) {
            const int pl = it / Q, q = it - pl * Q, n = L - 4 * q;
            const float* x = buf + pl * L + 4 * q;
            float4 r = make_float4(x[0], n > 1 ? x[1] : 0.0f, n > 2 ? x[2] : 0.0f, n > 3 ? x[3] : 0.0f);
            if (norm) {
                const float s = norm[p0 + pl];
                r.x = fmul(r.x, s);
                r.y = n > 1 ? fmul(r.y, s) : 0.0f;
                r.z = n > 2 ? fmul(r.z, s) : 0.0f;
                r.w = n > 3 ? fmul(r.w, s) : 0.0f;
            }
            rows[(p0 * Q) + it] = r;
        }
        __syncwarp();  // buf is refilled
    }
}

// The lists a splat launch covers: positions [first, first + count) of
// `order`, or the live images' positions of the domain behind lv.
struct SplatRange {
    int first = 0, count = 0;
    Live lv;
};
__device__ __forceinline__ int splat_vertex(const SplatRange& r, const int* __restrict__ order, long u) {
    return order[r.lv.n ? live_unit(r.lv, u) : r.first + u];
}

// Thread t of nt of the short lists' part.
template <int QC>
__device__ __forceinline__ void splat_rows_short(const SplatRange& r, int Qrt, const int* __restrict__ order,
                                                 const int* __restrict__ seg_start,
                                                 const int2* __restrict__ seg,
                                                 const float4* __restrict__ rows, float4* __restrict__ vals, long t0,
                                                 long nt) {
    const int Q = QC ? QC : Qrt;
    const long total = live_total(r.lv, r.count) * Q;
    for (long t = t0; t < total; t += nt) {
        const long u = t / Q;
        const int q = (int)(t - u * Q);
        const int v = splat_vertex(r, order, u);
        const int s0 = seg_start[v], s1 = seg_start[v + 1];
        unsigned long long a0 = 0ull, a1 = 0ull;
        // four entries per step, loaded two at a time from an even position
        // (those outside the list are not used)
        const int4* seg2 = reinterpret_cast<const int4*>(seg);
        int s = s0 & ~1;
        int4 ea, eb;
        if (s < s1) {
            ea = seg2[s >> 1];
            eb = seg2[(s >> 1) + 1];
        }
        for (; s < s1; s += kSplatU) {
            int p[kSplatU] = {ea.x, ea.z, eb.x, eb.z};
            const float w[kSplatU] = {__int_as_float(ea.y), __int_as_float(ea.w), __int_as_float(eb.y),
                                      __int_as_float(eb.w)};
            ulonglong2 x[kSplatU];
#pragma unroll
            for (int i = 0; i < kSplatU; i++) {  // no branch: the four loads go out together
                if (s + i < s0 || s + i >= s1) p[i] = 0;
                x[i] = *reinterpret_cast<const ulonglong2*>(rows + (long)p[i] * Q + q);
            }
            const int sn = (s + kSplatU < s1 ? s + kSplatU : s) >> 1;
            ea = seg2[sn];
            eb = seg2[sn + 1];
#pragma unroll
            for (int i = 0; i < kSplatU; i++)
                if (s + i >= s0 && s + i < s1) {
                    a0 = add_mul2(a0, w[i], x[i].x);
                    a1 = add_mul2(a1, w[i], x[i].y);
                }
        }
        *reinterpret_cast<ulonglong2*>(vals + (long)(v + 1) * Q + q) = make_ulonglong2(a0, a1);
    }
}

// The sum of one staged chunk of n <= E entries of rows of nq float4: this
// lane's label at xs, the weights at ws.
template <int E>
__device__ __forceinline__ float splat_sum_chunk(float acc, const float* xs, const float* ws, int nq, int n) {
    if (n == E) {
#pragma unroll
        for (int g = 0; g < E / 4; g++) {
            const float4 w = reinterpret_cast<const float4*>(ws)[g];
            acc = fadd(acc, fmul(w.x, xs[(4 * g + 0) * 4 * nq]));
            acc = fadd(acc, fmul(w.y, xs[(4 * g + 1) * 4 * nq]));
            acc = fadd(acc, fmul(w.z, xs[(4 * g + 2) * 4 * nq]));
            acc = fadd(acc, fmul(w.w, xs[(4 * g + 3) * 4 * nq]));
        }
    } else {
#pragma unroll 4
        for (int e = 0; e < n; e++) acc = fadd(acc, fmul(ws[e], xs[e * 4 * nq]));
    }
    return acc;
}

// Bytes of ring per warp for rows of nq float4 (at most 8 at a time).
__host__ __device__ constexpr int splat_ring_bytes(int nq) { return kSplatStages * 32 * (nq * 16 + 4); }

// Long lists: warp `unit0` of nw.
template <int QC>
__device__ __forceinline__ void splat_rows_long(const SplatRange& r, int Qrt, const int* __restrict__ order,
                                                const int* __restrict__ seg_start, const int2* __restrict__ seg, const float4* __restrict__ rows,
                                                float4* __restrict__ vals, unsigned char* ring, long unit0,
                                                long nw) {
    const int Q = QC ? QC : Qrt;
    const int lane = threadIdx.x & 31;
    const long total = live_total(r.lv, r.count);
    for (long unit = unit0; unit < total; unit += nw) {  // warp-uniform
        const int v = splat_vertex(r, order, unit);
        const int s0 = seg_start[v], s1 = seg_start[v + 1];
        const int nch = (s1 - s0 + 31) >> 5;
        for (int qb = 0; qb < Q; qb += 8) {  // 32 labels at a time
            const int nq = QC ? QC : min(8, Q - qb);
            float4* X = reinterpret_cast<float4*>(ring);                            // [stage][entry][nq]
            float* Wt = reinterpret_cast<float*>(X + kSplatStages * 32 * nq);       // [stage][entry]
            auto pix_of = [&](int c) {
                const int s = s0 + c * 32 + lane;
                return (c < nch && s < s1) ? seg[s].x : 0;
            };
            auto issue = [&](int c, int pc) {
                const int slot = c % kSplatStages, base = s0 + c * 32, n = min(32, s1 - base);
                if (lane < n) cp_async4(Wt + slot * 32 + lane, &seg[base + lane].y);
#pragma unroll
                for (int i = 0; i < (QC ? QC : 8); i++) {
                    if (!QC && i >= nq) break;
                    const int idx = lane + 32 * i, e = idx / nq;
                    const int p = __shfl_sync(0xffffffffu, pc, e);
                    if (e < n) cp_async16(X + slot * 32 * nq + idx, rows + (long)p * Q + qb + (idx - e * nq));
                }
            };
            float acc = 0.0f;
            int pcur = pix_of(0);
#pragma unroll
            for (int c = 0; c < kSplatStages - 1; c++) {
                const int pn = pix_of(c + 1);
                if (c < nch) issue(c, pcur);
                cp_async_commit();
                pcur = pn;
            }
            for (int c = 0; c < nch; c++) {
                const int ci = c + kSplatStages - 1;
                const int pn = pix_of(ci + 1);
                if (ci < nch) issue(ci, pcur);
                cp_async_commit();
                pcur = pn;
                cp_async_wait<kSplatStages - 1>();  // chunk c has landed (this lane's copies)
                __syncwarp();                       // ... and every other lane's
                const int slot = c % kSplatStages, n = min(32, s1 - (s0 + c * 32));
                if (lane < 4 * nq)
                    acc = splat_sum_chunk<32>(acc, reinterpret_cast<const float*>(X + slot * 32 * nq) + lane,
                                              Wt + slot * 32, nq, n);
                __syncwarp();  // the slot is refilled kSplatStages - 1 chunks later
            }
            cp_async_wait<0>();
            __syncwarp();
            if (lane < 4 * nq) reinterpret_cast<float*>(vals)[((long)(v + 1) * Q + qb) * 4 + lane] = acc;
        }
    }
}

// Huge lists: block b takes the b-th of the visiting order.
constexpr int kHugeE = 64;                              // entries per chunk
constexpr int kHugeStages = kSplatWarps * kSplatStages / 2;  // the four warps' rings as one
template <int QC>
__device__ __forceinline__ void splat_rows_huge(int b, int Qrt, const int* __restrict__ order,
                                                const int* __restrict__ seg_start, const int2* __restrict__ seg, const float4* __restrict__ rows,
                                                float4* __restrict__ vals, unsigned char* ring) {
    const int Q = QC ? QC : Qrt;
    const int t = threadIdx.x;
    constexpr int kMax = kHugeE * 8 / kSplatThreads;  // copies per thread and chunk, at most
    {
        const int v = order[b];
        const int s0 = seg_start[v], s1 = seg_start[v + 1];
        const int nch = (s1 - s0 + kHugeE - 1) / kHugeE;
        for (int qb = 0; qb < Q; qb += 8) {  // 32 labels at a time
            const int nq = QC ? QC : min(8, Q - qb);
            const int ncopy = kHugeE * nq;
            float4* X = reinterpret_cast<float4*>(ring);                        // [stage][entry][nq]
            float* Wt = reinterpret_cast<float*>(X + kHugeStages * ncopy);      // [stage][entry]
            // this thread's copies: entry (t + i threads) / nq of each chunk;
            // their pixels are loaded two chunks before their rows
            auto pix = [&](int c, int (&p)[kMax]) {
#pragma unroll
                for (int i = 0; i < kMax; i++) {
                    const int idx = t + i * kSplatThreads;
                    p[i] = -1;
                    if (idx < ncopy && c < nch) {
                        const int s = s0 + c * kHugeE + idx / nq;
                        if (s < s1) p[i] = seg[s].x;
                    }
                }
            };
            auto issue = [&](int c, const int (&p)[kMax]) {
                if (c < nch) {
                    const int slot = c % kHugeStages;
#pragma unroll
                    for (int i = 0; i < kMax; i++) {
                        const int idx = t + i * kSplatThreads;
                        if (idx < ncopy && p[i] >= 0)
                            cp_async16(X + slot * ncopy + idx, rows + (long)p[i] * Q + qb + idx % nq);
                    }
                    const int s = s0 + c * kHugeE + t;
                    if (t < kHugeE && s < s1) cp_async4(Wt + slot * kHugeE + t, &seg[s].y);
                }
                cp_async_commit();
            };
            int pa[kMax], pb[kMax];
            pix(0, pa);
            pix(1, pb);
            auto step = [&](int c) {  // chunk c's copies, then the pixels of chunk c + 2
                issue(c, pa);
#pragma unroll
                for (int i = 0; i < kMax; i++) pa[i] = pb[i];
                pix(c + 2, pb);
            };
#pragma unroll 1
            for (int c = 0; c < kHugeStages - 1; c++) step(c);
            float acc = 0.0f;
            for (int c = 0; c < nch; c++) {
                cp_async_wait<kHugeStages - 2>();  // chunk c has landed (this thread's copies)
                __syncthreads();                   // ... and everyone's; chunk c - 1 is summed
                step(c + kHugeStages - 1);
                if (t < 4 * nq) {
                    const int slot = c % kHugeStages;
                    acc = splat_sum_chunk<kHugeE>(acc, reinterpret_cast<const float*>(X + slot * ncopy) + t,
                                                  Wt + slot * kHugeE, nq, min(kHugeE, s1 - (s0 + c * kHugeE)));
                }
            }
            cp_async_wait<0>();
            __syncthreads();  // the ring is refilled
            if (t < 4 * nq) reinterpret_cast<float*>(vals)[((long)(v + 1) * Q + qb) * 4 + t] = acc;
        }
    }
}

// Blocks [0, huge_blocks) take the huge lists (the first of the visiting
// order, longest first, so that the longest chain starts at once), the next
// long_blocks the long ones and the others the short ones: one launch, the
// short lists filling the SMs that the long chains leave idle.  A lattice
// without long lists launches no such blocks and no shared memory.
// A block per huge list pays while those lists are few enough to be all
// resident and their chains set the launch's length (at most four per SM, a
// single image: 640x480 bilateral 50 -> 30 us); where there are more, and in
// batches, its one adding warp would leave the SMs idle (16 images of 512x512
// have some 4000: 345 us against 276) and they count as long lists.
constexpr int kHugePerSM = 4;
template <int QC>
__global__ void __launch_bounds__(kSplatThreads)
    splat_rows_kernel(SplatRange rl, SplatRange rs, int huge_blocks, int long_blocks, int Q,
                      const int* __restrict__ order, const int* __restrict__ seg_start,
                      const int2* __restrict__ seg,
                      const float4* __restrict__ rows, float4* __restrict__ vals, float4* __restrict__ other) {
    extern __shared__ __align__(16) unsigned char splat_smem[];
    grid_release();
    grid_wait();
    if (blockIdx.x == gridDim.x - 1)  // row 0 of both value buffers: what absent neighbours read
        for (int q = threadIdx.x; q < (QC ? QC : Q); q += blockDim.x)
            vals[q] = other[q] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    int b = blockIdx.x;
    if (b < huge_blocks) {
        splat_rows_huge<QC>(b, Q, order, seg_start, seg, rows, vals, splat_smem);
        return;
    }
    b -= huge_blocks;
    if (b < long_blocks) {
        const int wib = threadIdx.x >> 5;
        splat_rows_long<QC>(rl, Q, order, seg_start, seg, rows, vals,
                            splat_smem + wib * splat_ring_bytes(QC ? QC : min(Q, 8)), (long)b * kSplatWarps + wib,
                            (long)long_blocks * kSplatWarps);
        return;
    }
    b -= long_blocks;
    splat_rows_short<QC>(rs, Q, order, seg_start, seg, rows, vals, (long)b * blockDim.x + threadIdx.x,
                         (long)(gridDim.x - huge_blocks - long_blocks) * blockDim.x);
}

// The splat for L = 1, 2 (seqCompute; also every normalisation factor): the
// same split of lists.  A long list's warp forms 128 products at a time (lane
// = entry, the next 128 entries' values in flight) and lanes 0 .. L-1 add
// them in entry order from shared memory; a short list takes one thread per
// label.
constexpr int kThinE = 128;  // entries per step of a long list

template <int L>
__global__ void __launch_bounds__(kSplatThreads)
    splat_thin_kernel(SplatRange rl, SplatRange rs, int long_blocks, const int* __restrict__ order,
                      const int* __restrict__ seg_start, const int2* __restrict__ seg, const float* __restrict__ in, const float* __restrict__ norm,
                      float* __restrict__ vals, float* __restrict__ other) {
    __shared__ __align__(16) float prod[kSplatWarps][L][kThinE];
    constexpr int U = kThinE / 32;
    grid_release();
    grid_wait();
    if (blockIdx.x == 0 && threadIdx.x < L) vals[threadIdx.x] = other[threadIdx.x] = 0.0f;  // absent neighbours
    if ((int)blockIdx.x < long_blocks) {
        const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
        const long total = live_total(rl.lv, rl.count);
        for (long unit = (long)blockIdx.x * kSplatWarps + wib; unit < total;
             unit += (long)long_blocks * kSplatWarps) {  // warp-uniform
            const int v = splat_vertex(rl, order, unit);
            const int s0 = seg_start[v], s1 = seg_start[v + 1];
            int p[U];
            float w[U], wc[U], x[U][L];
            auto load_pw = [&](int c) {
#pragma unroll
                for (int i = 0; i < U; i++) {
                    const int s = min(c + i * 32 + lane, s1 - 1);
                    const int2 e = seg[s];
                    p[i] = e.x;
                    w[i] = entry_w(e);
                }
            };
            auto load_x = [&] {  // the values of the entries p, scaled; their weights become wc
#pragma unroll
                for (int i = 0; i < U; i++) {
                    const float nn = norm ? norm[p[i]] : 1.0f;
                    wc[i] = w[i];
#pragma unroll
                    for (int k = 0; k < L; k++) {
                        x[i][k] = in[(long)p[i] * L + k];
                        if (norm) x[i][k] = fmul(x[i][k], nn);
                    }
                }
            };
            load_pw(s0);
            load_x();
            load_pw(s0 + kThinE);  // past the end: the last entry again
            float acc = 0.0f;
            for (int c = s0; c < s1; c += kThinE) {
#pragma unroll
                for (int i = 0; i < U; i++)
#pragma unroll
                    for (int k = 0; k < L; k++) prod[wib][k][i * 32 + lane] = fmul(wc[i], x[i][k]);
                if (c + kThinE < s1) {  // in flight while this step is added
                    load_x();
                    load_pw(c + 2 * kThinE);
                }
                __syncwarp();
                if (lane < L) {
                    const int n = min(kThinE, s1 - c);
                    const float* pr = prod[wib][lane];
                    int e = 0;
                    for (; e + 16 <= n; e += 16) {
                        float4 q[4];
#pragma unroll
                        for (int g = 0; g < 4; g++) q[g] = reinterpret_cast<const float4*>(pr + e)[g];
#pragma unroll
                        for (int g = 0; g < 4; g++) {
                            acc = fadd(acc, q[g].x);
                            acc = fadd(acc, q[g].y);
                            acc = fadd(acc, q[g].z);
                            acc = fadd(acc, q[g].w);
                        }
                    }
                    for (; e < n; e++) acc = fadd(acc, pr[e]);
                }
                __syncwarp();  // prod is rewritten next step
            }
            if (lane < L) vals[(long)(v + 1) * L + lane] = acc;
        }
    } else {
        const long total = live_total(rs.lv, rs.count) * L;
        const long nt = (long)(gridDim.x - long_blocks) * blockDim.x;
        for (long t = (long)(blockIdx.x - long_blocks) * blockDim.x + threadIdx.x; t < total; t += nt) {
            const long u = t / L;
            const int k = (int)(t - u * L);
            const int v = splat_vertex(rs, order, u);
            const int s0 = seg_start[v], s1 = seg_start[v + 1];
            float acc = 0.0f;
            for (int s = s0; s < s1; s += 8) {
                float y[8];
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const int si = min(s + i, s1 - 1);
                    const int2 e = seg[si];
                    const int p = e.x;
                    float x = in[(long)p * L + k];
                    if (norm) x = fmul(x, norm[p]);
                    y[i] = fmul(entry_w(e), x);
                }
#pragma unroll
                for (int i = 0; i < 8; i++)
                    if (s + i < s1) acc = fadd(acc, y[i]);
            }
            vals[(long)(v + 1) * L + k] = acc;
        }
    }
}

__global__ void count_long_kernel(int M, const int* __restrict__ counts, int threshold, int* __restrict__ n) {
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    const bool is_long = v < M && counts[v] > threshold;
    const unsigned b = __ballot_sync(0xffffffffu, is_long);
    if ((threadIdx.x & 31) == 0 && b) atomicAdd(n, __popc(b));
}

// Class of a splat list by its length: 0 long, 1 short.
__device__ __forceinline__ int list_class(int c) { return c > kLongList ? 0 : 1; }

// Concatenated lattices: the key (class, image) of each position of the
// length-sorted visiting order, for a second stable sort that groups each
// class's lists by image (longest first within an image), and the number of
// lists per (class, image).
__global__ void class_image_key_kernel(int M, const int* __restrict__ order, const int* __restrict__ counts,
                                       const int* __restrict__ vimg, int images, int* __restrict__ keys,
                                       int* __restrict__ per_class_image) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= M) return;
    const int v = order[p];
    const int key = list_class(counts[v]) * images + vimg[v];
    keys[p] = key;
    atomicAdd(&per_class_image[key], 1);
}

// Sort key of the splat visiting order (stable radix sort ascending): the
// long lists first, longest first, so that their chains start early; the
// short lists after them in vertex-id order.  Ids follow the pixels' scan
// order (first occurrence), so consecutive short lists gather rows of nearby
// pixels and each input row is fetched from DRAM about once although d + 1
// lists read it (sorting the short lists by length too scattered them over
// the whole image).
__global__ void order_key_kernel(int M, const int* __restrict__ counts, int* __restrict__ keys,
                                 int* __restrict__ vals) {
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= M) return;
    const int c = counts[v];
    keys[v] = c > kLongList ? kMaxOrderKey - min(c, kMaxOrderKey) : kMaxOrderKey;
    vals[v] = v;
}

// One blur pass along one lattice axis: new = old + 1/2 (n1 + n2).  seqCompute
// evaluates it in double (0.5 is a double literal there, :518).
template <bool SEQ, int LC = 0>
__global__ void blur_kernel(int M, int Lrt, const int2* __restrict__ nbr,
                            const float* __restrict__ src, float* __restrict__ dst, Live lv) {
    const int L = LC ? LC : Lrt;
    grid_release();
    grid_wait();
    const long total = live_total(lv, M) * L;
    for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (long)gridDim.x * blockDim.x) {
        const long u = t / L;
        const int k = (int)(t - u * L);
        const int v = (int)live_unit(lv, u);
        const int2 nb = nbr[v];
        const float a = src[(long)(v + 1) * L + k];
        const float s = fadd(src[(long)nb.x * L + k], src[(long)nb.y * L + k]);
        float r;
        if (SEQ) r = (float)dadd((double)a, dmul(0.5, (double)s));
        else r = fadd(a, fmul(0.5f, s));
        dst[(long)(v + 1) * L + k] = r;
    }
}

// The blur pass over rows padded to Lp = 4 Q floats (sseCompute, L > 2):
// one thread per (vertex, four labels), float4 loads of the vertex's row and
// of its two neighbours' rows.  The same operations per element as
// blur_kernel; the padding lanes hold zeros and stay zero.
// SEQ: the half-sum in double, as blur_kernel<true> (the lattice gradient).
template <int Q, bool SEQ = false>
__global__ void blur4_kernel(int M, int Qrt, const int2* __restrict__ nbr, const float* __restrict__ src,
                             float* __restrict__ dst, Live lv) {
    const int Qn = Q ? Q : Qrt;
    const long lp = 4L * Qn;
    grid_release();
    grid_wait();
    const long total = live_total(lv, M) * Qn;
    for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (long)gridDim.x * blockDim.x) {
        const long u = t / Qn;
        const int q = (int)(t - u * Qn);
        const int v = (int)live_unit(lv, u);
        const int2 nb = nbr[v];
        const float4 a = *reinterpret_cast<const float4*>(src + (long)(v + 1) * lp + 4 * q);
        const float4 x = *reinterpret_cast<const float4*>(src + (long)nb.x * lp + 4 * q);
        const float4 y = *reinterpret_cast<const float4*>(src + (long)nb.y * lp + 4 * q);
        auto one = [](float c, float n1, float n2) {
            const float s = fadd(n1, n2);
            return SEQ ? (float)dadd((double)c, dmul(0.5, (double)s)) : fadd(c, fmul(0.5f, s));
        };
        const float4 r = make_float4(one(a.x, x.x, y.x), one(a.y, x.y, y.y), one(a.z, x.z, y.z), one(a.w, x.w, y.w));
        *reinterpret_cast<float4*>(dst + (long)(v + 1) * lp + 4 * q) = r;
    }
}

__device__ __forceinline__ float apply_epilogue(float v, long t, int i, int k, const SliceEpilogue& ep) {
    if (ep.potts) {
        if (ep.norm) v = fmul(v, ep.norm[i]);
        v = ep.scale_vec ? fmul(ep.scale_vec[k], v) : fmul(ep.scale, v);
    }
    if (ep.base) v = fadd(ep.base[t], fmul(ep.coef, v));
    else if (ep.zero_base) v = fadd(0.0f, fmul(ep.coef, v));
    return v;
}

// Slice: out(i, k) = sum_j (bary_ij * alpha) * value(o_ij, k) (sseCompute,
// :1046-1051) or sum_j (bary_ij * value) * alpha (seqCompute, :529-534).
template <bool SEQ, int DC, int LC>
__global__ void slice_kernel(int N, int Lrt, int drt, const int* __restrict__ offset,
                             const float* __restrict__ bary, const float* __restrict__ vals,
                             float alpha, float* out, SliceEpilogue ep, Live lv) {
    const int L = LC ? LC : Lrt, d = DC ? DC : drt;
    const int d1 = d + 1;
    grid_release();
    grid_wait();
    const long total = live_total(lv, N) * L;
    for (long tl = (long)blockIdx.x * blockDim.x + threadIdx.x; tl < total; tl += (long)gridDim.x * blockDim.x) {
        const long u = tl / L;
        const int k = (int)(tl - u * L);
        const int i = (int)live_unit(lv, u);  // the pixel
        const long t = (long)i * L + k;
        float acc = 0.0f;
#pragma unroll
        for (int j = 0; j <= d; j++) {
            const int o = offset[(long)i * d1 + j];
            const float w = bary[(long)i * d1 + j];
            const float v = vals[(long)(o + 1) * L + k];
            if (SEQ) acc = fadd(acc, fmul(fmul(w, v), alpha));
            else acc = fadd(acc, fmul(fmul(w, alpha), v));
        }
        out[t] = apply_epilogue(acc, t, i, k, ep);
    }
}

// Slice over rows of Q float4 (sseCompute, L > 2), a tile of pixels per warp
// (no block barrier: the warps' loads overlap each other's sums).  The tile's
// (row, barycentric * alpha) pairs and normalisation factors are staged in
// shared memory and the accumulation base (out = base + coef * v) is copied
// there asynchronously meanwhile; then lane (p, q) -- for L = 21 five pixels of
// six 16-byte groups per instruction -- gathers its pixel's d+1 vertex rows
// with 16-byte loads, applies the epilogue and leaves its four labels in shared
// memory, and the tile, contiguous in `out`, is stored with 16-byte accesses
// where the pointers allow (vec).  Per element the arithmetic is
// slice_kernel's and apply_epilogue's: acc = sum over j in order of (bary_j *
// alpha) * value_j, from +0.
// DOT: `out` is not written; the warp's FP64 sum of dot[e] * v[e] goes to
// partials[warp] instead.
constexpr int kSliceWarps = 4;
constexpr int kSliceTile = 20;  // pixels per warp tile (4 rounds of 5 at L = 21)
template <int DC, int Q, int LC, bool DOT>
__global__ void __launch_bounds__(32 * kSliceWarps)
    slice_rows_kernel(int N, int Lrt, int Qrt, int drt, int tile, const int* __restrict__ offset,
                      const float* __restrict__ bary, const float4* __restrict__ vals, float alpha, float* out,
                      SliceEpilogue ep, Live lv, const long* __restrict__ pix_base, int vec,
                      const float* __restrict__ dot, double* __restrict__ partials) {
    extern __shared__ __align__(16) unsigned char slice_smem[];
    const int d1 = (DC ? DC : drt) + 1, Qn = Q ? Q : Qrt, L = LC ? LC : Lrt;
    const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tf = (tile * L + 3) & ~3;  // floats of the output tile
    unsigned char* mine = slice_smem + (size_t)wib * ((tf * 4 + tile * (d1 * 8 + 8) + 15) & ~15);
    float* s_out = reinterpret_cast<float*>(mine);               // [tile][L]
    int2* s_ow = reinterpret_cast<int2*>(s_out + tf);            // [tile][d1]
    float* s_nrm = reinterpret_cast<float*>(s_ow + tile * d1);   // [tile]
    const bool use_norm = ep.potts && ep.norm;
    const float* base = DOT ? dot : ep.base;
    const int ppr = Qn <= 32 ? 32 / Qn : 1;       // pixels per round (Qn <= 32)
    const int lp = Qn <= 32 ? lane / Qn : 0;      // this lane's pixel of the round
    const int q0 = Qn <= 32 ? lane - lp * Qn : lane;
    double g = 0.0;
    grid_release();
    grid_wait();
    // Tiles: of the whole pixel range, or (live images) of each live image's
    // pixels, image by image (pix_base: its pixel offsets).
    const long total = live_total(lv, ((long)N + tile - 1) / tile);
    for (long u = (long)blockIdx.x * kSliceWarps + wib; u < total; u += (long)gridDim.x * kSliceWarps) {
        long p0;
        const int np = tile_pixels(lv, pix_base, u, tile, N, p0);
        const long t0 = p0 * L;
        const int ne = np * L;
        const int n4 = vec && (t0 & 3) == 0 ? ne >> 2 : 0;  // whole 16-byte groups of the tile
        if (base) {
            for (int e = lane; e < n4; e += 32) cp_async16(s_out + 4 * e, base + t0 + 4 * e);
            for (int e = 4 * n4 + lane; e < ne; e += 32) cp_async4(s_out + e, base + t0 + e);
        }
        cp_async_commit();
        for (int e = lane; e < np * d1; e += 32)
            s_ow[e] = make_int2((offset[p0 * d1 + e] + 1) * Qn, __float_as_int(fmul(bary[p0 * d1 + e], alpha)));
        if (use_norm)
            for (int e = lane; e < np; e += 32) s_nrm[e] = ep.norm[p0 + e];
        cp_async_wait<0>();
        __syncwarp();
        auto item = [&](int pl, int q) {
            const int2* ow = s_ow + pl * d1;
            const float4* vq = vals + q;
            unsigned long long a0 = 0ull, a1 = 0ull;
            auto add = [&](int2 e) {
                const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(vq + e.x);
                const float wa = __int_as_float(e.y);
                a0 = add_mul2(a0, wa, v.x);
                a1 = add_mul2(a1, wa, v.y);
            };
            if (DC) {
#pragma unroll
                for (int j = 0; j < DC + 1; j++) add(ow[j]);
            } else {
                for (int j = 0; j < d1; j++) add(ow[j]);
            }
            const float2 lo = unpack2(a0), hi = unpack2(a1);
            float v[4] = {lo.x, lo.y, hi.x, hi.y};
            const int k0 = 4 * q;
            float* so = s_out + pl * L + k0;
            if (use_norm) {
                const float nn = s_nrm[pl];
#pragma unroll
                for (int c = 0; c < 4; c++) v[c] = fmul(v[c], nn);
            }
            if (ep.potts) {
                if (ep.scale_vec) {
#pragma unroll
                    for (int c = 0; c < 4; c++)
                        if (k0 + c < L) v[c] = fmul(ep.scale_vec[k0 + c], v[c]);
                } else {
#pragma unroll
                    for (int c = 0; c < 4; c++) v[c] = fmul(ep.scale, v[c]);
                }
            }
            if (DOT) {
#pragma unroll
                for (int c = 0; c < 4; c++)
                    if (k0 + c < L) g += (double)so[c] * (double)v[c];
                return;
            }
            if (base) {
#pragma unroll
                for (int c = 0; c < 4; c++)
                    if (k0 + c < L) so[c] = fadd(so[c], fmul(ep.coef, v[c]));
            } else {
#pragma unroll
                for (int c = 0; c < 4; c++)
                    if (k0 + c < L) so[c] = ep.zero_base ? fadd(0.0f, fmul(ep.coef, v[c])) : v[c];
            }
        };
        if (Qn <= 32) {
            if (lp < ppr) {
#pragma unroll 2
                for (int pl = lp; pl < np; pl += ppr) item(pl, q0);
            }
        } else {
            for (int pl = 0; pl < np; pl++)
                for (int q = q0; q < Qn; q += 32) item(pl, q);
        }
        __syncwarp();
        if (DOT) {
            __syncwarp();
        } else {
            float4* o4 = reinterpret_cast<float4*>(out + t0);
            for (int e = lane; e < n4; e += 32) o4[e] = reinterpret_cast<const float4*>(s_out)[e];
            for (int e = 4 * n4 + lane; e < ne; e += 32) out[t0 + e] = s_out[e];
            __syncwarp();  // the next tile restages the shared arrays
        }
    }
    if (DOT) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) g += __shfl_down_sync(0xffffffffu, g, o);
        if (lane == 0) partials[(long)blockIdx.x * kSliceWarps + wib] = g;
    }
}

// addSplitArray / sliceSplitArray bins (:548-589): the lower pass rounds
// q*10 in float, the upper pass (q - 1e-9)*10 in double.
// For q in [0, 1] these are the reference's indices; other values (which the
// reference rejects with an assert) are clamped to a valid bin so no access
// can leave the bin array.
__device__ __forceinline__ int bin_lower(float q) {
    int c = (int)floorf(fmul(q, (float)kRes));
    c = c < kRes - 1 ? c : kRes - 1;
    return c > 0 ? c : 0;
}
__device__ __forceinline__ int bin_upper(float q) {
    int c = (int)floor(dmul(__dsub_rn((double)q, 1e-9), (double)kRes));
    c = c > 0 ? c : 0;
    return c < kRes - 1 ? c : kRes - 1;
}

// Ordered bins of every (pixel, label), computed once per ordered filter
// (each pixel appears in d+1 splat lists and in the slice): the lower and
// upper bin indices, held as floats (exact small integers) because the splat
// compares them with float bin numbers.
__device__ __forceinline__ float2 ord_bin_pair(float q) {
    return make_float2((float)bin_lower(q), (float)bin_upper(q));
}
__device__ __forceinline__ int ord_lower_of(float2 b) { return (int)b.x; }
__device__ __forceinline__ int ord_upper_of(float2 b) { return (int)b.y; }

__global__ void ord_bins_kernel(long n, const float* __restrict__ Q, float2* __restrict__ bins) {
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    bins[t] = ord_bin_pair(Q[t]);
}

// The same, four elements per thread with 16-byte loads and stores (Q and
// bins 16-byte aligned; n4 = n / 4 quads, the tail by ord_bins_kernel).
__global__ void ord_bins4_kernel(long n4, const float4* __restrict__ Q, float4* __restrict__ bins) {
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n4) return;
    const float4 q = Q[t];
    const float2 a = ord_bin_pair(q.x), b = ord_bin_pair(q.y), c = ord_bin_pair(q.z), d = ord_bin_pair(q.w);
    bins[2 * t] = make_float4(a.x, a.y, b.x, b.y);
    bins[2 * t + 1] = make_float4(c.x, c.y, d.x, d.y);
}

// Each of the 10 bins accumulates, in entry order, the weights of the entries
// that reach it: bins 0..c (lower pass) or c..9 (upper pass), addSplitArray
// (:548-569).  Branch-free and bit-identical: the mask m = [c_lower >= b]
// (lower) or [b >= c_upper] (upper) is exactly 1.0 or 0.0 (one PTX `set`,
// NaN giving 0), so fma(m, w, acc) rounds acc + w once when the entry reaches
// the bin and otherwise returns acc (acc + (+-0) = acc: the accumulator
// starts at +0 and is never -0).
__device__ __forceinline__ float step_ge(float a, float b) {  // a >= b ? 1 : 0
    float r;
    asm("set.ge.f32.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

// One entry into the bin-b pair (lower, upper) of packed accumulators:
// acc = fma({[cl >= b], [b >= cu]}, w2, acc) with one f32x2 FMA, which rounds
// each half exactly as fma.rn.f32 does.  w2 holds (w, w).  The bins are
// small integers, so the masks are saturated sums: cl + (1 - b) and
// (b + 1) - cu are exact integers, clamped to [0, 1] they are exactly the
// comparisons (and a NaN would clamp to +0).  One `add.sat` per mask.
__device__ __forceinline__ void ord_step2(unsigned long long& acc, float cl, float cu, float b,
                                          unsigned long long w2) {
    const float lo_c = 1.0f - b, up_c = b + 1.0f;  // exact; hoisted out of the entry loops
    asm("{\n\t.reg .f32 ml, mu;\n\t.reg .b64 m;\n\t"
        "add.rn.sat.f32 ml, %1, %3;\n\t"
        "sub.rn.sat.f32 mu, %4, %2;\n\t"
        "mov.b64 m, {ml, mu};\n\t"
        "fma.rn.f32x2 %0, m, %5, %0;\n\t}"
        : "+l"(acc)
        : "f"(cl), "f"(cu), "f"(lo_c), "f"(up_c), "l"(w2));
}
// The single masks of ord_step2: [cl >= b] and [b >= cu] as 0.0 / 1.0.
__device__ __forceinline__ float ord_mask_lower(float cl, int b) {
    float m;
    asm("add.rn.sat.f32 %0, %1, %2;" : "=f"(m) : "f"(cl), "f"(1.0f - (float)b));
    return m;
}
__device__ __forceinline__ float ord_mask_upper(float cu, int b) {
    float m;
    asm("sub.rn.sat.f32 %0, %1, %2;" : "=f"(m) : "f"((float)b + 1.0f), "f"(cu));
    return m;
}
template <bool UPPER>
__device__ __forceinline__ void ord_accumulate(float (&acc)[kRes], float c, float w) {
#pragma unroll
    for (int b = 0; b < kRes; b++) {
        const float m = UPPER ? step_ge((float)b, c) : step_ge(c, (float)b);
        acc[b] = __fmaf_rn(m, w, acc[b]);
    }
}

template <bool UPPER>
__device__ __forceinline__ void ord_consume(float (&acc)[kRes], const float (*ring)[32], const float* mw, int lane,
                                            int n) {
#pragma unroll 2
    for (int e = 0; e < n; e++) ord_accumulate<UPPER>(acc, ring[e][lane], mw[e]);
}

// Ordered splat, general L: one warp per (vertex, pass), streaming the
// vertex's list as splat_kernel does.  A vertex row holds 20 bins x L
// labels, bin-major ([v][bin][label]; bins [0,10) lower, [10,20) upper) so
// that the slice's per-label bin reads coalesce.
__global__ void __launch_bounds__(32 * kStageWarps)
    ord_splat_kernel(int M, int L, const int* __restrict__ order, const int* __restrict__ seg_start,
                     const int2* __restrict__ seg,
                     const float2* __restrict__ bins, float* __restrict__ vals) {
    __shared__ float ring[kStageWarps][kStages][kChunk][32];
    __shared__ float mw[kStageWarps][kStages][kChunk];
    const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int unit = blockIdx.x * kStageWarps + wib;
    if (unit >= 2 * M) return;  // warp-uniform
    const int v = order[unit >> 1];
    const bool upper = unit & 1;
    const int s0 = seg_start[v], s1 = seg_start[v + 1];
    const float* bf = reinterpret_cast<const float*>(bins);  // [pixel][label][lower, upper]
    for (int kb = 0; kb < L; kb += 32) {
        const int k = kb + lane;
        const bool act = k < L;
        float acc[kRes];
#pragma unroll
        for (int b = 0; b < kRes; b++) acc[b] = 0.0f;
        stream_list<float>(s0, s1, 2 * L, 2 * k + (upper ? 1 : 0), act, lane, seg, bf, ring[wib], mw[wib],
                           [&](int slot, int n) {
                               if (upper) ord_consume<true>(acc, ring[wib][slot], mw[wib][slot], lane, n);
                               else ord_consume<false>(acc, ring[wib][slot], mw[wib][slot], lane, n);
                           });
        if (act) {
            float* row = vals + ((long)(v + 1) * kOrdW + (upper ? kRes : 0)) * L + k;
#pragma unroll
            for (int b = 0; b < kRes; b++) row[(long)b * L] = acc[b];
        }
    }
}

// Ordered splat of the long lists by blocks.  The 20 x L bin sums of a
// vertex are 20 L independent in-order chains; thread (k, g) carries the
// chains of label k, bins g*NB .. g*NB+NB-1, both passes, so a block shares
// a long list's work and the longest lists no longer set the kernel's
// length.
//
// The list streams through shared memory in chunks of kOE entries: the
// pixel ids and weights of chunk c + 2 kODX and the (c_lower, c_upper) bins
// of chunk c + kODX are copied with cp.async while chunk c is summed, one
// block barrier per chunk.  Ring rows are label-major ([k][entry][lower,
// upper], padded to an odd number of 16-byte units) so a thread reads two
// entries per 16-byte load and eight consecutive labels hit distinct banks.
// Weights are staged as (w, w) pairs; entries past the end of the list get
// weight 0, which leaves every accumulator unchanged (the masks are 0 or 1
// for any stale bin value).
constexpr int kOE = 32;                 // entries per chunk
constexpr int kODX = 4;                 // bins are copied kODX chunks ahead of use, pixel ids 2 kODX
constexpr int kOXS = kODX + 1;          // bin ring slots (chunks c .. c+kODX)
constexpr int kOPS = 2 * kODX + 1;      // pixel / weight ring slots (chunks c .. c+2 kODX)
constexpr int kORow = 2 * kOE + 4;      // floats per ring row: 17 x 16 bytes
constexpr int kOrdBlockMaxL = 160;      // larger L use ord_splat_kernel (shared-memory ring size)
constexpr int kGroupChoices[] = {1, 2, 3, 5, 10};

// Bin split with the fewest warp instructions per list entry: warps x (three
// instructions per bin slot -- two masks and one f32x2 FMA -- + about two
// for the shared-memory loads).
int ord_groups_cheapest(int L) {
    int best = 1;
    long best_cost = -1;
    for (int G : kGroupChoices) {
        if (L * G > 1024) break;
        const long warps = (L * G + 31) / 32, nb = (kRes + G - 1) / G;
        const long cost = warps * (3 * nb + 2);
        if (best_cost < 0 || cost <= best_cost) {
            best = G;
            best_cost = cost;
        }
    }
    return best;
}

size_t ord_block_smem(int kb) {
    return sizeof(float) * ((size_t)kOXS * kb * kORow + (size_t)kOPS * kOE * 2) + sizeof(int) * kOPS * kOE;
}

// G bin groups per label, NB = ceil(10 / G) bin slots per thread; slots past
// bin 9 (when G does not divide 10) run on a dummy bin that is not stored.
// Block b covers labels [k0, k0 + nk) of vertex order[b / kblocks], k0 =
// (b % kblocks) * kb: a very long list can be shared by several blocks.
// Compute threads are label-major (t = k * G + g), so the G threads reading
// one label's bins sit in one warp and their shared-memory loads broadcast;
// staging threads are entry-major (t = g * nk + k) so one warp's copies read
// consecutive labels of one pixel.
template <int G>
__global__ void __launch_bounds__(kOrdBlockMaxL * G < 1024 ? kOrdBlockMaxL * G : 1024)
    ord_splat_block_kernel(int L, int kb, int kblocks, const int* __restrict__ order,
                           const int* __restrict__ seg_start, const int2* __restrict__ seg, const float2* __restrict__ bins,
                           float* __restrict__ vals) {
    extern __shared__ __align__(16) float osm[];
    float* xr = osm;                            // [kOXS][kb][kORow]
    float* wr = xr + (size_t)kOXS * kb * kORow;  // [kOPS][kOE][2]
    int* pr = reinterpret_cast<int*>(wr + kOPS * kOE * 2);  // [kOPS][kOE]
    constexpr int NB = (kRes + G - 1) / G;
    const int t = threadIdx.x;
    const int v = order[blockIdx.x / kblocks];
    const int k0 = (blockIdx.x % kblocks) * kb, nk = min(kb, L - k0);
    const int s0 = seg_start[v], s1 = seg_start[v + 1];
    const int nch = (s1 - s0 + kOE - 1) / kOE;
    const bool worker = t < nk * G;
    const int k = t / G, g = t - k * G;      // compute role
    const int sk = t % nk, sg = t / nk;      // staging role (sg < G for workers)

    auto stage_pw = [&](int c) {  // pixel ids and weights of chunk c
        if (c < nch && t < kOE) {
            const int slot = c % kOPS, e = s0 + c * kOE + t;
            if (e < s1) {
                cp_async4(&pr[slot * kOE + t], &seg[e].x);
                cp_async4(&wr[(slot * kOE + t) * 2], &seg[e].y);
                cp_async4(&wr[(slot * kOE + t) * 2 + 1], &seg[e].y);
            } else {
                pr[slot * kOE + t] = 0;
                wr[(slot * kOE + t) * 2] = 0.0f;
                wr[(slot * kOE + t) * 2 + 1] = 0.0f;
            }
        }
    };
    // (c_lower, c_upper) of chunk c; needs chunk c's pixel ids in place.
    // Staging thread (sk, sg) copies label k0 + sk of entries sg, sg + G, ...
    // All pixel ids are read before the first copy is issued (the copies'
    // memory clobber would otherwise order each read after the last copy).
    auto stage_x = [&](int c) {
        if (c >= nch || !worker) return;
        constexpr int MX = (kOE + G - 1) / G;
        const int slot = c % kOXS, ps = c % kOPS;
        const int n = min(kOE, s1 - (s0 + c * kOE));
        float* dst = &xr[((size_t)slot * kb + sk) * kORow];
        const float2* src = bins + k0 + sk;
        int pix[MX];
#pragma unroll
        for (int i = 0; i < MX; i++) {
            const int e = sg + i * G;
            pix[i] = e < n ? pr[ps * kOE + e] : 0;
        }
#pragma unroll
        for (int i = 0; i < MX; i++) {
            const int e = sg + i * G;
            if (e < n) cp_async8(dst + 2 * e, src + (long)pix[i] * L);
        }
    };

    // Group j (committed at iteration j; j < 0 in the prologue) holds the
    // bins of chunk j + kODX and the pixel ids / weights of chunk j + 2 kODX.
#pragma unroll
    for (int c = 0; c < kODX; c++) stage_pw(c);
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
#pragma unroll
    for (int c = 0; c < kODX; c++) {
        stage_x(c);
        stage_pw(c + kODX);
        cp_async_commit();
    }

    // Bin g*NB + i's (lower, upper) sums as one packed pair: ord_step2 adds
    // an entry to both with one f32x2 FMA (each half rounded as fma.rn.f32).
    unsigned long long acc[NB];
    float bf[NB];
#pragma unroll
    for (int i = 0; i < NB; i++) {
        acc[i] = 0ull;
        bf[i] = (float)(g * NB + i);
    }
    for (int c = 0; c < nch; c++) {
        cp_async_wait<kODX - 1>();  // group c - kODX: bins of chunk c, pixel ids of chunk c + kODX
        __syncthreads();            // ... everyone's copies; and chunk c-1's slots are free
        stage_x(c + kODX);
        stage_pw(c + 2 * kODX);
        cp_async_commit();
        if (worker) {
            const float4* xs = reinterpret_cast<const float4*>(&xr[((size_t)(c % kOXS) * kb + k) * kORow]);
            const ulonglong2* ws = reinterpret_cast<const ulonglong2*>(&wr[(c % kOPS) * kOE * 2]);
            const int n2 = (min(kOE, s1 - (s0 + c * kOE)) + 1) >> 1;
            // Batches of eight entries, the next batch's loads issued before
            // this batch is summed.  A batch may run past n2 into the chunk's
            // zero-weight tail (the ring rows hold kOE entries).
            float4 x[4];      // (c_lower, c_upper) of entries 2 j, 2 j + 1
            ulonglong2 w[4];  // ((w, w), (w, w)) of the same entries
#pragma unroll
            for (int j = 0; j < 4; j++) {
                x[j] = xs[j];
                w[j] = ws[j];
            }
            for (int b0 = 0; b0 < n2; b0 += 4) {
                float4 xn[4];
                ulonglong2 wn[4];
                const int nb0 = b0 + 4 < kOE / 2 ? b0 + 4 : b0;  // stays inside the ring row
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    xn[j] = xs[nb0 + j];
                    wn[j] = ws[nb0 + j];
                }
#pragma unroll
                for (int j = 0; j < 4; j++) {
#pragma unroll
                    for (int i = 0; i < NB; i++) ord_step2(acc[i], x[j].x, x[j].y, bf[i], w[j].x);
#pragma unroll
                    for (int i = 0; i < NB; i++) ord_step2(acc[i], x[j].z, x[j].w, bf[i], w[j].y);
                }
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    x[j] = xn[j];
                    w[j] = wn[j];
                }
            }
        }
    }
    cp_async_wait<0>();
    if (worker) {
        float* row = vals + (long)(v + 1) * kOrdW * L + k0 + k;
#pragma unroll
        for (int i = 0; i < NB; i++) {
            if (g * NB + i >= kRes) break;
            const float2 r = unpack2(acc[i]);
            row[(long)(g * NB + i) * L] = r.x;
            row[(long)(kRes + g * NB + i) * L] = r.y;
        }
    }
}

// Ordered splat of the short lists: one thread per (vertex, label), both
// passes, without staging.
template <int LC = 0>
__global__ void ord_splat_short_kernel(int n_short, int Lrt, const int* __restrict__ order,
                                       const int* __restrict__ seg_start, const int2* __restrict__ seg, const float2* __restrict__ bins,
                                       float* __restrict__ vals) {
    const int L = LC ? LC : Lrt;
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long)n_short * L) return;
    const int u = (int)(t / L), k = (int)(t - (long)u * L);
    const int v = order[u];
    const int s0 = seg_start[v], s1 = seg_start[v + 1];
    // Scalar chains: every entry reaches lower bin 0 (c_lower >= 0) and upper
    // bin 9 (c_upper <= 9), plain adds there; the other 18 bins take a
    // saturated-sum mask (exactly 0 or 1) and an FMA, fma(1, w, acc) being
    // acc + w rounded once.
    float lo[kRes], up[kRes];
#pragma unroll
    for (int b = 0; b < kRes; b++) lo[b] = up[b] = 0.0f;
#pragma unroll 2
    for (int s = s0; s < s1; s++) {
        const float2 x = bins[(long)seg[s].x * L + k];
        const float w = entry_w(seg[s]);
        lo[0] = fadd(lo[0], w);
#pragma unroll
        for (int b = 1; b < kRes; b++) lo[b] = __fmaf_rn(ord_mask_lower(x.x, b), w, lo[b]);
#pragma unroll
        for (int b = 0; b < kRes - 1; b++) up[b] = __fmaf_rn(ord_mask_upper(x.y, b), w, up[b]);
        up[kRes - 1] = fadd(up[kRes - 1], w);
    }
    float* row = vals + (long)(v + 1) * kOrdW * L + k;
#pragma unroll
    for (int b = 0; b < kRes; b++) {
        row[(long)b * L] = lo[b];
        row[(long)(kRes + b) * L] = up[b];
    }
}

// Ordered blur: every bin independently, weightedAddSplitArray (:570-578).
template <int R4>  // row width in float4 as a compile-time constant (0 = run-time row4r)
__global__ void ord_blur_kernel(int M, int row4r, const int2* __restrict__ nbr,
                                const float4* __restrict__ src, float4* __restrict__ dst) {
    const int row4 = R4 ? R4 : row4r;
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long)M * row4) return;
    const int v = (int)(t / row4), c = (int)(t - (long)v * row4);
    const int2 nb = nbr[v];
    const float4 a = src[(long)(v + 1) * row4 + c];
    const float4 p = src[(long)nb.x * row4 + c];
    const float4 q = src[(long)nb.y * row4 + c];
    float4 r;
    r.x = fadd(a.x, fmul(0.5f, fadd(p.x, q.x)));
    r.y = fadd(a.y, fmul(0.5f, fadd(p.y, q.y)));
    r.z = fadd(a.z, fmul(0.5f, fadd(p.z, q.z)));
    r.w = fadd(a.w, fmul(0.5f, fadd(p.w, q.w)));
    dst[(long)(v + 1) * row4 + c] = r;
}

// Ordered slice: lower pass with weight -w*alpha, then upper with w*alpha
// (:639-650, :687-696), accumulated into one value.  With GAP the LP's dual
// gap terms are folded in: tmp = (alpha + u) - (v + su) for the final slice
// value v, the clique term su (0 without cliques), and per-block sums of
// tmp.Q and tmp.tmp (src/densecrf.cpp:725-729).
// DC / LC: d and L as compile-time constants (0 = run-time drt / Lrt).
template <bool GAP, int DC, int LC>
__global__ void __launch_bounds__(kTB, 8) ord_slice_kernel(int N, int Lrt, int drt, const int* __restrict__ offset,
                                 const float* __restrict__ bary, const float* __restrict__ vals,
                                 const float2* __restrict__ bins, float alpha, float* out, SliceEpilogue ep,
                                 GapFusion gf) {
    const int L = LC ? LC : Lrt, d = DC ? DC : drt;
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    double g0 = 0.0, g1 = 0.0;
    if (t < (long)N * L) {
        const int i = (int)(t / L), k = (int)(t - (long)i * L);
        const int d1 = d + 1;
        const float2 bp = bins[t];
        const int cl = ord_lower_of(bp), cu = ord_upper_of(bp);
        float acc = 0.0f;
#pragma unroll
        for (int j = 0; j <= d; j++) {
            const int o = offset[(long)i * d1 + j];
            const float w = bary[(long)i * d1 + j];
            acc = fadd(acc, fmul(vals[((long)(o + 1) * kOrdW + cl) * L + k], fmul(-w, alpha)));
        }
#pragma unroll
        for (int j = 0; j <= d; j++) {
            const int o = offset[(long)i * d1 + j];
            const float w = bary[(long)i * d1 + j];
            acc = fadd(acc, fmul(vals[((long)(o + 1) * kOrdW + kRes + cu) * L + k], fmul(w, alpha)));
        }
        const float v = apply_epilogue(acc, t, i, k, ep);
        out[t] = v;
        if (GAP) {
            const float tmp = fsub(fadd(gf.alpha[t], gf.u[t]), fadd(v, gf.su ? gf.su[t] : 0.0f));
            g0 = (double)tmp * (double)gf.Q[t];
            g1 = (double)tmp * (double)tmp;
        }
    }
    if (GAP) {
        __shared__ double s0[kTB / 32], s1[kTB / 32];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            g0 += __shfl_down_sync(0xffffffffu, g0, o);
            g1 += __shfl_down_sync(0xffffffffu, g1, o);
        }
        if ((threadIdx.x & 31) == 0) {
            s0[threadIdx.x >> 5] = g0;
            s1[threadIdx.x >> 5] = g1;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            double a = 0.0, b = 0.0;
            for (int w = 0; w < kTB / 32; w++) {
                a += s0[w];
                b += s1[w];
            }
            gf.partials[blockIdx.x] = a;
            gf.partials[gridDim.x + blockIdx.x] = b;
        }
    }
}

// One term of a fused two-term ordered slice.
struct OrdSliceTerm {
    const int* offset;
    const float* bary;
    const float* vals;
    int d;
    float alpha;
    SliceEpilogue ep;
};

template <int DC>
__device__ __forceinline__ float ord_slice_acc(const OrdSliceTerm& s, int i, int k, int L, int cl, int cu) {
    const int d = DC ? DC : s.d, d1 = d + 1;
    const int* __restrict__ off = s.offset + (long)i * d1;
    const float* __restrict__ by = s.bary + (long)i * d1;
    float acc = 0.0f;
#pragma unroll
    for (int j = 0; j <= d; j++)
        acc = fadd(acc, fmul(s.vals[((long)(off[j] + 1) * kOrdW + cl) * L + k], fmul(-by[j], s.alpha)));
#pragma unroll
    for (int j = 0; j <= d; j++)
        acc = fadd(acc, fmul(s.vals[((long)(off[j] + 1) * kOrdW + kRes + cu) * L + k], fmul(by[j], s.alpha)));
    return acc;
}

// sa = t1's slice on top of t0's (Model::apply_ord_sum with two terms): v0 =
// epilogue_0(slice_0) exactly as ord_slice_kernel writes it, then v0 +
// coef_1 * scaled(slice_1) as ord_slice_kernel computes it from base = v0.
// The value v0 never leaves the register; GAP as in ord_slice_kernel.
template <bool GAP, int D0, int D1, int LC>
__global__ void __launch_bounds__(kTB, 8) ord_slice_pair_kernel(int N, int Lrt, OrdSliceTerm t0, OrdSliceTerm t1,
                                      const float2* __restrict__ bins, float* out, GapFusion gf) {
    const int L = LC ? LC : Lrt;
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    double g0 = 0.0, g1 = 0.0;
    if (t < (long)N * L) {
        const int i = (int)(t / L), k = (int)(t - (long)i * L);
        const float2 bp = bins[t];
        const int cl = ord_lower_of(bp), cu = ord_upper_of(bp);
        const float a0 = ord_slice_acc<D0>(t0, i, k, L, cl, cu);
        const float a1 = ord_slice_acc<D1>(t1, i, k, L, cl, cu);
        const float v0 = apply_epilogue(a0, t, i, k, t0.ep);
        float s1 = a1;
        if (t1.ep.potts) {
            if (t1.ep.norm) s1 = fmul(s1, t1.ep.norm[i]);
            s1 = t1.ep.scale_vec ? fmul(t1.ep.scale_vec[k], s1) : fmul(t1.ep.scale, s1);
        }
        const float v = fadd(v0, fmul(t1.ep.coef, s1));
        out[t] = v;
        if (GAP) {
            const float tmp = fsub(fadd(gf.alpha[t], gf.u[t]), fadd(v, gf.su ? gf.su[t] : 0.0f));
            g0 = (double)tmp * (double)gf.Q[t];
            g1 = (double)tmp * (double)tmp;
        }
    }
    if (GAP) {
        __shared__ double s0[kTB / 32], s1[kTB / 32];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            g0 += __shfl_down_sync(0xffffffffu, g0, o);
            g1 += __shfl_down_sync(0xffffffffu, g1, o);
        }
        if ((threadIdx.x & 31) == 0) {
            s0[threadIdx.x >> 5] = g0;
            s1[threadIdx.x >> 5] = g1;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            double a = 0.0, b = 0.0;
            for (int w = 0; w < kTB / 32; w++) {
                a += s0[w];
                b += s1[w];
            }
            gf.partials[blockIdx.x] = a;
            gf.partials[gridDim.x + blockIdx.x] = b;
        }
    }
}

// ord_slice_pair_kernel for the LP's common case (L = 21, a d = 2 and a
// d = 5 term) with the per-pixel data staged: a block covers the same 256
// elements (at most 14 pixels), and its pixels' offsets, alpha-scaled
// barycentric weights and normalisation factors are loaded once, coalesced,
// into shared memory instead of by each label's thread.  Element, block and
// dual-gap partial sums are those of ord_slice_pair_kernel, so the values
// are too: the lower pass's fmul(-w, alpha) is the exact negation of
// fmul(w, alpha).
template <bool GAP>
__global__ void __launch_bounds__(kTB, 8) ord_slice_pair_staged(int N, OrdSliceTerm t0, OrdSliceTerm t1,
                                                               const float2* __restrict__ bins, float* out,
                                                               GapFusion gf) {
    constexpr int L = 21, D0 = 3, D1 = 6, P = kTB / L + 2;  // pixels a block touches at most
    __shared__ int so0[P * D0], so1[P * D1];
    __shared__ float sw0[P * D0], sw1[P * D1], sn0[P], sn1[P];
    const long NL = (long)N * L;
    const long tb = (long)blockIdx.x * blockDim.x;
    const long t = tb + threadIdx.x;
    const int pf = (int)(tb / L);
    const int np = (int)min((long)P, (long)N - pf);
    for (int e = threadIdx.x; e < np * D0; e += blockDim.x) {
        so0[e] = t0.offset[(long)pf * D0 + e];
        sw0[e] = fmul(t0.bary[(long)pf * D0 + e], t0.alpha);
    }
    for (int e = threadIdx.x; e < np * D1; e += blockDim.x) {
        so1[e] = t1.offset[(long)pf * D1 + e];
        sw1[e] = fmul(t1.bary[(long)pf * D1 + e], t1.alpha);
    }
    if (threadIdx.x < np) {
        if (t0.ep.norm) sn0[threadIdx.x] = t0.ep.norm[pf + threadIdx.x];
        if (t1.ep.norm) sn1[threadIdx.x] = t1.ep.norm[pf + threadIdx.x];
    }
    __syncthreads();
    double g0 = 0.0, g1 = 0.0;
    if (t < NL) {
        const int i = (int)(t / L), k = (int)(t - (long)i * L), li = i - pf;
        const float2 bp = bins[t];
        const int cl = ord_lower_of(bp), cu = ord_upper_of(bp);
        float a0 = 0.0f, a1 = 0.0f;
#pragma unroll
        for (int j = 0; j < D0; j++)
            a0 = fadd(a0, fmul(t0.vals[((long)(so0[li * D0 + j] + 1) * kOrdW + cl) * L + k], -sw0[li * D0 + j]));
#pragma unroll
        for (int j = 0; j < D0; j++)
            a0 = fadd(a0, fmul(t0.vals[((long)(so0[li * D0 + j] + 1) * kOrdW + kRes + cu) * L + k], sw0[li * D0 + j]));
#pragma unroll
        for (int j = 0; j < D1; j++)
            a1 = fadd(a1, fmul(t1.vals[((long)(so1[li * D1 + j] + 1) * kOrdW + cl) * L + k], -sw1[li * D1 + j]));
#pragma unroll
        for (int j = 0; j < D1; j++)
            a1 = fadd(a1, fmul(t1.vals[((long)(so1[li * D1 + j] + 1) * kOrdW + kRes + cu) * L + k], sw1[li * D1 + j]));
        float v0 = a0;
        if (t0.ep.potts) {
            if (t0.ep.norm) v0 = fmul(v0, sn0[li]);
            v0 = t0.ep.scale_vec ? fmul(t0.ep.scale_vec[k], v0) : fmul(t0.ep.scale, v0);
        }
        if (t0.ep.base) v0 = fadd(t0.ep.base[t], fmul(t0.ep.coef, v0));
        else if (t0.ep.zero_base) v0 = fadd(0.0f, fmul(t0.ep.coef, v0));
        float s1 = a1;
        if (t1.ep.potts) {
            if (t1.ep.norm) s1 = fmul(s1, sn1[li]);
            s1 = t1.ep.scale_vec ? fmul(t1.ep.scale_vec[k], s1) : fmul(t1.ep.scale, s1);
        }
        const float v = fadd(v0, fmul(t1.ep.coef, s1));
        out[t] = v;
        if (GAP) {
            const float tmp = fsub(fadd(gf.alpha[t], gf.u[t]), fadd(v, gf.su ? gf.su[t] : 0.0f));
            g0 = (double)tmp * (double)gf.Q[t];
            g1 = (double)tmp * (double)tmp;
        }
    }
    if (GAP) {
        __shared__ double s0[kTB / 32], s1[kTB / 32];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            g0 += __shfl_down_sync(0xffffffffu, g0, o);
            g1 += __shfl_down_sync(0xffffffffu, g1, o);
        }
        if ((threadIdx.x & 31) == 0) {
            s0[threadIdx.x >> 5] = g0;
            s1[threadIdx.x >> 5] = g1;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            double a = 0.0, b = 0.0;
            for (int w = 0; w < kTB / 32; w++) {
                a += s0[w];
                b += s1[w];
            }
            gf.partials[blockIdx.x] = a;
            gf.partials[gridDim.x + blockIdx.x] = b;
        }
    }
}

// Bins of rescale(Q) (src/eigen_utils.cpp:120-141) without materialising it:
// rq = (Q - min) / (max - min), with min / max at qmm[0], qmm[1].
__global__ void rescaled_bins_kernel(long n, const float* __restrict__ Q, const float* __restrict__ qmm,
                                     float2* __restrict__ bins) {
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const float mn = qmm[0], range = fsub(qmm[1], qmm[0]);
    float rq = fsub(Q[t], mn);
    if (range > 0.0f) rq = rq / range;
    bins[t] = ord_bin_pair(rq);
}

// The same, four elements per thread (as ord_bins4_kernel).
__global__ void rescaled_bins4_kernel(long n4, const float4* __restrict__ Q, const float* __restrict__ qmm,
                                      float4* __restrict__ bins) {
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n4) return;
    const float mn = qmm[0], range = fsub(qmm[1], qmm[0]);
    const float4 q = Q[t];
    float r[4] = {fsub(q.x, mn), fsub(q.y, mn), fsub(q.z, mn), fsub(q.w, mn)};
    if (range > 0.0f)
#pragma unroll
        for (int i = 0; i < 4; i++) r[i] = r[i] / range;
    const float2 a = ord_bin_pair(r[0]), b = ord_bin_pair(r[1]), c = ord_bin_pair(r[2]), d = ord_bin_pair(r[3]);
    bins[2 * t] = make_float4(a.x, a.y, b.x, b.y);
    bins[2 * t + 1] = make_float4(c.x, c.y, d.x, d.y);
}

bool aligned16(const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }

// Ordered-filter bins of Q [n]: four per thread where the pointers allow.
void ord_bins(float2* bins, const float* Q, long n, cudaStream_t st) {
    if (aligned16(Q) && aligned16(bins)) {
        const long n4 = n / 4;
        if (n4) launch(ord_bins4_kernel, ceil_div(n4, kTB), kTB, 0, st, n4, reinterpret_cast<const float4*>(Q),
                       reinterpret_cast<float4*>(bins));
        if (n > 4 * n4) launch(ord_bins_kernel, 1, kTB, 0, st, n - 4 * n4, Q + 4 * n4, bins + 4 * n4);
    } else {
        launch(ord_bins_kernel, ceil_div(n, kTB), kTB, 0, st, n, Q, bins);
    }
}

int bits_for(int n) {  // bits needed to hold values 0..n-1
    int b = 0;
    while ((1LL << b) < (long long)n) b++;
    return b;
}

template <int DM>
void build_impl(Lattice& L, const float* d_features) {
    constexpr int KW = (DM + 7) / 8;
    cudaStream_t st = L.stream;
    const int N = L.N, d = L.d, d1 = d + 1;
    const int Np = (N + 3) & ~3;
    const long E = (long)Np * d1, Ereal = (long)N * d1;
    require(E < (1L << 30), DCRF_E_ARG, "lattice too large (N*(d+1) >= 2^30)");

    // scale_factor (:190-194): computed in double, rounded to float.
    std::vector<float> scale(d);
    const float inv_std_dev = (float)(std::sqrt(2.0 / 3.0) * (d + 1));
    for (int i = 0; i < d; i++) scale[i] = (float)(1.0 / std::sqrt((double)((i + 2) * (i + 1))) * inv_std_dev);
    float* dscale = L.fscale.ensure(d);
    DCRF_CUDA(cudaMemcpyAsync(dscale, scale.data(), sizeof(float) * d, cudaMemcpyHostToDevice, st));

    int4* ekeys = L.ekeys.ensure((size_t)E * KW);
    int* rank = L.rank.ensure(Ereal);
    float* bary = L.bary.ensure(Ereal);
    launch(elevate_kernel<DM>, ceil_div(Np, kTB), kTB, 0, st, d_features, N, Np, d, dscale, ekeys, rank, bary);
    DCRF_LAUNCH_CHECK();

    unsigned cap = 1;
    while ((long)cap < 2 * E) cap <<= 1;
    int* table = L.table.ensure(cap);
    DCRF_CUDA(cudaMemsetAsync(table, 0xff, sizeof(int) * cap, st));
    int* eslot = L.entry_slot.ensure(E);
    launch(insert_kernel<KW>, ceil_div(E, kTB), kTB, 0, st, ekeys, (int)E, table, cap - 1, eslot);
    int* flags = L.flags.ensure(E);
    launch(first_flag_kernel, ceil_div(E, kTB), kTB, 0, st, (int)E, eslot, table, flags);
    DCRF_LAUNCH_CHECK();
    int* dtotal = L.total.ensure(1);
    exclusive_scan(flags, flags, (int)E, dtotal, L.scan, st);
    int M = 0;
    DCRF_CUDA(cudaMemcpyAsync(&M, dtotal, sizeof(int), cudaMemcpyDeviceToHost, st));
    DCRF_CUDA(cudaStreamSynchronize(st));
    L.M = M;

    int* offset = L.offset.ensure(Ereal);
    int16_t* vkeys = L.vkeys.ensure((size_t)M * d);
    int* slot_vid = L.slot_vid.ensure(cap);
    launch(finalize_kernel<KW>, ceil_div(E, kTB), kTB, 0, st, (int)E, (int)Ereal, d, eslot, table, flags,
                                                         ekeys, offset, vkeys, slot_vid);
    int2* nbr = L.nbr.ensure((size_t)d1 * M);
    launch(neighbor_kernel<KW>, ceil_div((long)d1 * M, kTB), kTB, 0, st, M, d, vkeys, table, cap - 1,
                                                                     ekeys, slot_vid, nbr);
    DCRF_LAUNCH_CHECK();

    // Splat lists: per-vertex counts -> starts; stable sort of entries by vertex.
    int* counts = L.counts.ensure((size_t)M + 1);
    DCRF_CUDA(cudaMemsetAsync(counts, 0, sizeof(int) * ((size_t)M + 1), st));
    launch(count_kernel, ceil_div(Ereal, kTB), kTB, 0, st, (int)Ereal, offset, counts);
    int* seg_start = L.seg_start.ensure((size_t)M + 1);
    exclusive_scan(counts, seg_start, M + 1, nullptr, L.scan, st);
    int* skeys = L.sort_keys.ensure(Ereal);
    int* svals = L.sort_vals.ensure(Ereal);
    launch(iota_copy_kernel, ceil_div(Ereal, kTB), kTB, 0, st, (int)Ereal, offset, skeys, svals);
    DCRF_LAUNCH_CHECK();
    radix_sort_pairs(skeys, svals, (int)Ereal, bits_for(M), L.sort, st);
    int2* seg = L.seg.ensure(Ereal + kSegPad);
    launch(seg_fill_kernel, ceil_div(Ereal, kTB), kTB, 0, st, (int)Ereal, d1, svals, bary, seg);
    // Splat visiting order: longest lists first.
    int* vorder = L.vorder.ensure(M);
    int* okeys = L.vorder_keys.ensure(M);
    launch(order_key_kernel, ceil_div(M, kTB), kTB, 0, st, M, counts, okeys, vorder);
    radix_sort_pairs(okeys, vorder, M, 24, L.sort, st);
    int* dlong = L.total.ensure(2);
    DCRF_CUDA(cudaMemsetAsync(dlong, 0, 2 * sizeof(int), st));
    launch(count_long_kernel, ceil_div(M, kTB), kTB, 0, st, M, counts, kLongList, dlong);
    launch(count_long_kernel, ceil_div(M, kTB), kTB, 0, st, M, counts, kHugeList, dlong + 1);
    DCRF_LAUNCH_CHECK();
    int nl[2];
    DCRF_CUDA(cudaMemcpyAsync(nl, dlong, 2 * sizeof(int), cudaMemcpyDeviceToHost, st));
    DCRF_CUDA(cudaStreamSynchronize(st));
    L.n_long = nl[0];
    L.n_huge = nl[1];
    L.va_floats = 0;
}

}  // namespace

// Row stride of the plain filter's value buffers: L padded to a multiple of
// four (float4 rows) on the sseCompute path (L > 2); seqCompute (L <= 2)
// keeps L.
static int value_row(int L) { return L > 2 ? (L + 3) & ~3 : L; }

// Blocks of a launch over `units` work items, `per_block` per block of
// `threads` threads: all of them at once, or -- with live images, whose
// units are counted on the device -- twice as many blocks as the SMs hold
// at full occupancy, looping over them.
static int unit_grid(long units, int per_block, bool live, int threads) {
    const long g = std::max(1L, (units + per_block - 1) / per_block);
    return live ? (int)std::min(g, (long)sm_count() * 2 * (2048 / threads)) : (int)g;
}

namespace {

// ----------------------------------------------------- feature gradient --
// Permutohedral::gradient (src/permutohedral.cpp:1095-1178): df [N][d] of
// a^T K b with respect to the (scaled) features.  For each direction the
// host splats one side, blurs with the double-evaluated 1/2 weights in axis
// order (reversed for the second direction), and this kernel forms the
// slice-side derivative per pixel in the reference's float order: for each
// label k, r_j = (0 + alpha v(o0_j)) - alpha v(o1_j) with o0/o1 from the
// pixel's ranks, then for j = 1..d, grad_j += x_k * sf_{j-1} (s - j r_j),
// s += r_j, s starting at r_0; finally df += grad.
struct GradScale {
    float s[16];
};

template <int DM>
__global__ void grad_slice_kernel(int N, int L, int Lp, int d, const int* __restrict__ offset, const int* __restrict__ rank,
                                  const float* __restrict__ vals, const float* __restrict__ x, float alpha,
                                  GradScale sf, float* __restrict__ df) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    const int d1 = d + 1;
    int o0[DM + 1], o1[DM + 1];
#pragma unroll
    for (int j = 0; j <= DM; j++)
        if (j <= d) {
            const int r0 = d - rank[(long)i * d1 + j];
            const int r1 = r0 + 1 > d ? 0 : r0 + 1;
            o0[j] = offset[(long)i * d1 + r0] + 1;
            o1[j] = offset[(long)i * d1 + r1] + 1;
        }
    float grad[DM];
#pragma unroll
    for (int j = 0; j < DM; j++) grad[j] = 0.0f;
    for (int k = 0; k < L; k++) {
        float ra[DM + 1];
#pragma unroll
        for (int j = 0; j <= DM; j++)
            if (j <= d)
                ra[j] = fsub(fadd(0.0f, fmul(alpha, vals[(long)o0[j] * Lp + k])), fmul(alpha, vals[(long)o1[j] * Lp + k]));
        const float xk = x[(long)i * L + k];
        float sm = ra[0];
#pragma unroll
        for (int j = 1; j <= DM; j++)
            if (j <= d) {
                const float v = fmul(sf.s[j - 1], fsub(sm, fmul((float)j, ra[j])));
                grad[j - 1] = fadd(grad[j - 1], fmul(xk, v));
                sm = fadd(sm, ra[j]);
            }
    }
#pragma unroll
    for (int j = 0; j < DM; j++)
        if (j < d) df[(long)i * d + j] = fadd(df[(long)i * d + j], grad[j]);
}

template <int DM>
void gradient_impl(Lattice& lat, float* df, const float* a, const float* b, int L) {
    cudaStream_t st = lat.stream;
    const int N = lat.N, d = lat.d, M = lat.M;
    const int Lp = value_row(L), Q = Lp / 4;
    lat.ensure_values((size_t)Lp);
    DCRF_CUDA(cudaMemsetAsync(df, 0, sizeof(float) * (size_t)N * d, st));
    // scale_factor and alpha as the reference computes them (:1104-1111)
    GradScale sf{};
    const float inv_std_dev = std::sqrt(2.0 / 3.0) * (d + 1);
    for (int i = 0; i < d; i++) sf.s[i] = 1.0 / std::sqrt(double((i + 2) * (i + 1))) * inv_std_dev;
    const float alpha = 1.0f / (1 + std::pow(2.0f, (float)-d)) / (d + 1);
    const long ML = (long)M * L, MQ = (long)M * Q;
    for (int dir = 0; dir < 2; dir++) {
        const float* in = dir ? b : a;
        float *src = lat.va.get(), *dst = lat.vb.get();
        lat.splat(in, L, nullptr, src);
        for (int jj = 0; jj <= d; jj++) {
            const int j = dir ? d - jj : jj;
            const int2* nb = lat.nbr.get() + (long)j * M;
            if (L <= 2) launch_chained(blur_kernel<true>, ceil_div(ML, kTB), kTB, 0, st, M, L, nb, src, dst, Live{});
            else if (Q == 6) launch_chained(blur4_kernel<6, true>, ceil_div(MQ, kTB), kTB, 0, st, M, Q, nb, src, dst, Live{});
            else launch_chained(blur4_kernel<0, true>, ceil_div(MQ, kTB), kTB, 0, st, M, Q, nb, src, dst, Live{});
            std::swap(src, dst);
        }
        launch(grad_slice_kernel<DM>, ceil_div(N, 128), 128, 0, st, N, L, Lp, d, lat.offset.get(), lat.rank.get(), src,
               dir ? a : b, alpha, sf, df);
    }
    DCRF_LAUNCH_CHECK();
}

}  // namespace

void Lattice::gradient(float* df, const float* a, const float* b, int L) {
    require(L >= 1, DCRF_E_ARG, "gradient: L must be >= 1");
    require(!concatenated, DCRF_E_STATE, "gradient: not available on a concatenated lattice");
    if (d <= 2) gradient_impl<2>(*this, df, a, b, L);
    else if (d <= 5) gradient_impl<5>(*this, df, a, b, L);
    else if (d <= 8) gradient_impl<8>(*this, df, a, b, L);
    else gradient_impl<16>(*this, df, a, b, L);
}

// ------------------------------------------------------ concatenation --
// Several images' lattices as one: vertex, pixel and entry ids of part i are
// shifted by the parts before it, so one filter launch sequence runs every
// image at once and each image's values are those of its own lattice (no
// list, neighbour or slice crosses an image).
namespace {

__global__ void add_offset_kernel(long n, const int* __restrict__ src, int add, int* __restrict__ dst) {
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) dst[t] = src[t] + add;
}

__global__ void seg_offset_kernel(long n, const int2* __restrict__ src, int add, int2* __restrict__ dst) {
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) dst[t] = make_int2(src[t].x + add, src[t].y);
}

// Neighbour rows are vertex + 1, with 0 for "absent".
__global__ void nbr_offset_kernel(long n, const int2* __restrict__ src, int add, int2* __restrict__ dst) {
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const int2 a = src[t];
    dst[t] = make_int2(a.x > 0 ? a.x + add : 0, a.y > 0 ? a.y + add : 0);
}

__global__ void fill_int_kernel(long n, int v, int* __restrict__ x) {
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) x[t] = v;
}

__global__ void seg_count_kernel(int M, const int* __restrict__ seg_start, int* __restrict__ counts) {
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v < M) counts[v] = seg_start[v + 1] - seg_start[v];
}

}  // namespace

void Lattice::concat(const std::vector<const Lattice*>& parts) {
    require(!parts.empty(), DCRF_E_ARG, "lattice concat: no parts");
    cudaStream_t st = stream;
    d = parts[0]->d;
    const int d1 = d + 1;
    long Nt = 0, Mt = 0;
    for (const Lattice* p : parts) {
        require(p->d == d, DCRF_E_ARG, "lattice concat: parts differ in feature dimension");
        Nt += p->N;
        Mt += p->M;
    }
    require(Nt * d1 < (1L << 30) && Mt < (1L << 30), DCRF_E_ARG, "lattice concat: too large");
    N = (int)Nt;
    M = (int)Mt;
    const long E = Nt * d1;
    int* off = offset.ensure(E);
    int* rk = rank.ensure(E);
    float* by = bary.ensure(E);
    int* ss = seg_start.ensure(M + 1);
    int2* sg = seg.ensure(E + kSegPad);
    int2* nb = nbr.ensure((size_t)d1 * M);
    int* vi = vimg.ensure(std::max(M, 1));
    long pb = 0, vb_ = 0;
    int part = 0;
    for (const Lattice* p : parts) {
        const long e = (long)p->N * d1, eb = pb * d1;
        DCRF_CUDA(cudaStreamSynchronize(p->stream));  // the part was built on its own stream
        launch(add_offset_kernel, ceil_div(e, kTB), kTB, 0, st, e, p->offset.get(), (int)vb_, off + eb);
        DCRF_CUDA(cudaMemcpyAsync(rk + eb, p->rank.get(), sizeof(int) * e, cudaMemcpyDeviceToDevice, st));
        DCRF_CUDA(cudaMemcpyAsync(by + eb, p->bary.get(), sizeof(float) * e, cudaMemcpyDeviceToDevice, st));
        if (p->M) {
            launch(add_offset_kernel, ceil_div(p->M, kTB), kTB, 0, st, (long)p->M, p->seg_start.get(), (int)eb,
                   ss + vb_);
            for (int j = 0; j < d1; j++)
                launch(nbr_offset_kernel, ceil_div(p->M, kTB), kTB, 0, st, (long)p->M,
                       p->nbr.get() + (long)j * p->M, (int)vb_, nb + (long)j * M + vb_);
        }
        launch(seg_offset_kernel, ceil_div(e, kTB), kTB, 0, st, e, (const int2*)p->seg.get(), (int)pb, sg + eb);
        if (p->M) launch(fill_int_kernel, ceil_div(p->M, kTB), kTB, 0, st, (long)p->M, part, vi + vb_);
        pb += p->N;
        vb_ += p->M;
        part++;
    }
    const int Ei = (int)E;
    DCRF_CUDA(cudaMemcpyAsync(ss + M, &Ei, sizeof(int), cudaMemcpyHostToDevice, st));
    // Longest lists first, over all images.
    int* cnt = counts.ensure(std::max(M, 1));
    launch(seg_count_kernel, ceil_div(M, kTB), kTB, 0, st, M, ss, cnt);
    int* vo = vorder.ensure(M);
    int* ok = vorder_keys.ensure(M);
    launch(order_key_kernel, ceil_div(M, kTB), kTB, 0, st, M, cnt, ok, vo);
    radix_sort_pairs(ok, vo, M, 24, sort, st);
    // Then, stably, by (class, image): each class (long, short lists) holds
    // its lists image by image, longest first within an image, so
    // that an image's lists of a class are one contiguous range of the order
    // (the live-image domains of a batched solve).
    const int B = (int)parts.size();
    DevBuf<int> pci;
    int* per_ci = pci.ensure((size_t)2 * B);
    DCRF_CUDA(cudaMemsetAsync(per_ci, 0, sizeof(int) * 2 * B, st));
    launch(class_image_key_kernel, ceil_div(M, kTB), kTB, 0, st, M, (const int*)vo, (const int*)cnt,
           (const int*)vi, B, ok, per_ci);
    int kbits = 1;
    while ((1L << kbits) < 2L * B) kbits++;
    radix_sort_pairs(ok, vo, M, kbits, sort, st);
    int* dl = total.ensure(2);
    DCRF_CUDA(cudaMemsetAsync(dl, 0, 2 * sizeof(int), st));
    launch(count_long_kernel, ceil_div(M, kTB), kTB, 0, st, M, cnt, kLongList, dl);
    launch(count_long_kernel, ceil_div(M, kTB), kTB, 0, st, M, cnt, kHugeList, dl + 1);
    DCRF_LAUNCH_CHECK();
    int nl[2];
    std::vector<int> hci((size_t)2 * B);
    DCRF_CUDA(cudaMemcpyAsync(nl, dl, 2 * sizeof(int), cudaMemcpyDeviceToHost, st));
    DCRF_CUDA(cudaMemcpyAsync(hci.data(), per_ci, sizeof(int) * 2 * B, cudaMemcpyDeviceToHost, st));
    DCRF_CUDA(cudaStreamSynchronize(st));  // also keeps &Ei alive until its copy ran
    n_long = nl[0];
    n_huge = nl[1];
    // Per-image domains: list positions per class, vertex ids, pixels.
    images = B;
    img_pixels.assign(B, 0);
    std::vector<long> hb((size_t)kDomains * (B + 1), 0);
    auto row = [&](int dom) { return hb.data() + (long)dom * (B + 1); };
    long pos = 0;
    for (int c = 0; c < 2; c++) {
        long* r = row(kDomLong + c);
        for (int i = 0; i < B; i++) {
            r[i] = pos;
            pos += hci[(size_t)c * B + i];
        }
        r[B] = pos;
    }
    for (int i = 0; i < B; i++) {
        img_pixels[i] = parts[i]->N;
        row(kDomVert)[i + 1] = row(kDomVert)[i] + parts[i]->M;
        row(kDomPix)[i + 1] = row(kDomPix)[i] + parts[i]->N;
    }
    long* db = dom_base.ensure(hb.size());
    DCRF_CUDA(cudaMemcpyAsync(db, hb.data(), sizeof(long) * hb.size(), cudaMemcpyHostToDevice, st));
    DCRF_CUDA(cudaStreamSynchronize(st));  // hb is the copy's source
    dom_tile = 0;
    va_floats = 0;
    concatenated = true;
}

void Lattice::prepare_live(int L) {
    require(concatenated && images > 0, DCRF_E_STATE, "live images: not a concatenated lattice");
    if (L <= 2) return;  // the element-wise slice needs no tile domain
    const int tile = slice_tile_for(L);
    if (tile == dom_tile) return;
    std::vector<long> r(images + 1, 0);
    for (int i = 0; i < images; i++) r[i + 1] = r[i] + (img_pixels[i] + tile - 1) / tile;
    DCRF_CUDA(cudaMemcpyAsync(dom_base.get() + (long)kDomTile * (images + 1), r.data(), sizeof(long) * r.size(),
                              cudaMemcpyHostToDevice, stream));
    DCRF_CUDA(cudaStreamSynchronize(stream));  // r is the copy's source
    dom_tile = tile;
}

void Lattice::build(const float* d_features, int d_, int N_) {
    require(N_ > 0, DCRF_E_ARG, "lattice: N must be positive");
    require(d_ >= 1 && d_ <= 16, DCRF_E_ARG, "lattice: feature dimension must be in [1, 16]");
    N = N_;
    d = d_;
    if (d <= 2) build_impl<2>(*this, d_features);
    else if (d <= 5) build_impl<5>(*this, d_features);
    else if (d <= 8) build_impl<8>(*this, d_features);
    else build_impl<16>(*this, d_features);
}

void Lattice::ensure_aux() {
    if (aux) return;
    int lo = 0, hi = 0;
    DCRF_CUDA(cudaDeviceGetStreamPriorityRange(&lo, &hi));
    DCRF_CUDA(cudaStreamCreateWithPriority(&aux, cudaStreamNonBlocking, hi));
    DCRF_CUDA(cudaEventCreateWithFlags(&ev_fork, cudaEventDisableTiming));
    DCRF_CUDA(cudaEventCreateWithFlags(&ev_join, cudaEventDisableTiming));
}

Lattice::~Lattice() {
    if (aux) {
        cudaStreamSynchronize(aux);
        cudaEventDestroy(ev_fork);
        cudaEventDestroy(ev_join);
        cudaStreamDestroy(aux);
    }
}

void Lattice::ensure_values(size_t row_width) {
    const size_t need = (size_t)(M + 1) * row_width;
    if (need > va_floats) {
        va.ensure(need);
        vb.ensure(need);
        va_floats = need;
    }
}

// ---------------------------------------------------------------------------
// Allocation-free filtering (dcrf_lattice_compute_noalloc).
//
// Some callers cannot let a library allocate device memory during a call:
// hosts that hand out all GPU memory from their own pool, or that run under a
// fixed memory budget in a latency-critical loop where a driver allocation
// would stall or fail.  For them the filter's two value buffers, normally
// grown on demand with cudaMalloc, come from this fixed array instead.  Every
// GPU that loads the library keeps it for the life of the process.
constexpr size_t kNoAllocScratchFloats = size_t(8) << 20;  // 8 Mi floats = 32 MiB
static __device__ __align__(256) float g_noalloc_scratch[kNoAllocScratchFloats];

namespace {
constexpr int kMaxDevices = 64;
std::mutex g_noalloc_mu;
float* g_noalloc_ptr[kMaxDevices] = {};

// Device address of the scratch array on the current device.  In host code
// the array's name is only a host-side stand-in, so the address is looked up
// once per device with that device current and cached.
float* noalloc_scratch() {
    int dev = 0;
    DCRF_CUDA(cudaGetDevice(&dev));
    require(dev >= 0 && dev < kMaxDevices, DCRF_E_ARG, "device index out of range");
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (!g_noalloc_ptr[dev]) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess)
            throw Error(DCRF_E_CUDA, std::string("cudaGetSymbolAddress(scratch): ") + cudaGetErrorString(e));
        g_noalloc_ptr[dev] = static_cast<float*>(p);
    }
    return g_noalloc_ptr[dev];
}
}  // namespace

size_t noalloc_scratch_floats() { return kNoAllocScratchFloats; }

void Lattice::compute_noalloc(float* out, const float* in, int L, bool reverse) {
    require(N > 0, DCRF_E_STATE, "lattice not initialised");
    require(L >= 1, DCRF_E_ARG, "compute: L must be >= 1");
    const size_t need = 2 * (size_t)(M + 1) * (size_t)L;
    require(need <= kNoAllocScratchFloats, DCRF_E_ARG,
            "compute_noalloc: 2 x (M + 1) x L = " + std::to_string(need) + " floats exceeds the fixed scratch of " +
                std::to_string(kNoAllocScratchFloats) + " floats (32 MiB); use dcrf_lattice_compute_dev");
    float* base = noalloc_scratch();
    float *src = base, *dst = base + (size_t)(M + 1) * L;
    cudaStream_t st = stream;
    // The array keeps the previous call's contents: only the zero rows that
    // absent neighbours read must be cleared; every other row read below is
    // written first.
    DCRF_CUDA(cudaMemsetAsync(src, 0, sizeof(float) * L, st));
    DCRF_CUDA(cudaMemsetAsync(dst, 0, sizeof(float) * L, st));
    const long ML = (long)M * L, NL = (long)N * L;
    const int n_short = M - n_long;
    if (n_long)
        launch(splat_kernel, ceil_div(n_long, kStageWarps), 32 * kStageWarps, 0, st, n_long, L, vorder.get(),
               seg_start.get(), seg.get(), in, src);
    if (n_short)
        launch(splat_short_kernel, ceil_div((long)n_short * L, kTB), kTB, 0, st, n_short, L,
               (const int*)vorder.get() + n_long, seg_start.get(), seg.get(), in, src);
    const bool seq = L <= 2;
    for (int jj = 0; jj <= d; jj++) {
        const int j = reverse ? d - jj : jj;
        if (seq)
            launch(blur_kernel<true>, ceil_div(ML, kTB), kTB, 0, st, M, L, nbr.get() + (long)j * M, src, dst, Live{});
        else
            launch(blur_kernel<false>, ceil_div(ML, kTB), kTB, 0, st, M, L, nbr.get() + (long)j * M, src, dst, Live{});
        std::swap(src, dst);
    }
    const float alpha = 1.0f / (1.0f + std::pow(2.0f, (float)-d));
    const SliceEpilogue ep;
    if (seq)
        launch(slice_kernel<true, 0, 0>, ceil_div(NL, kTB), kTB, 0, st, N, L, d, offset.get(), bary.get(), src, alpha,
               out, ep, Live{});
    else
        launch(slice_kernel<false, 0, 0>, ceil_div(NL, kTB), kTB, 0, st, N, L, d, offset.get(), bary.get(), src, alpha,
               out, ep, Live{});
    DCRF_LAUNCH_CHECK();
}

void Lattice::compute(float* out, const float* in, int L, bool reverse, const SliceEpilogue& ep,
                      const float* pre_norm) {
    splat_blur(in, L, reverse, pre_norm);
    slice(out, L, ep);
}

// Shared memory of the tiled slice: at most 10 KB per warp.
constexpr int kSliceSmem = 10 << 10;
static size_t slice_warp_bytes(int tile, int d, int L) {
    return ((size_t)((tile * L + 3) & ~3) * 4 + (size_t)tile * ((d + 1) * 8 + 8) + 15) & ~(size_t)15;
}
static int slice_tile_max(int tile, int d, int L) {
    while (tile > 1 && slice_warp_bytes(tile, d, L) > (size_t)kSliceSmem) tile = tile > 4 ? (tile / 2) & ~3 : tile - 1;
    return tile;
}

// Splats `in` [N][L] (times pre_norm) into vals: rows of Q float4 (L > 2) or
// of L floats.  With live images only their lists (and pixels).
void Lattice::splat(const float* in, int L, const float* pre_norm, float* vals) {
    cudaStream_t st = stream;
    const bool live = live_n != nullptr;
    const int n_short = M - n_long;
    const SplatRange rs{n_long, n_short, live_of(kDomShort)};
    float* other = vals == va.get() ? vb.get() : va.get();
    if (L <= 2) {
        const SplatRange rl{0, n_long, live_of(kDomLong)};
        const int lb = n_long ? unit_grid(n_long, kSplatWarps, live, kSplatThreads) : 0;
        const int sb = n_short ? unit_grid((long)n_short * L, kSplatThreads, live, kSplatThreads) : 0;
        if (lb + sb)
            launch_chained(L == 1 ? splat_thin_kernel<1> : splat_thin_kernel<2>, lb + sb, kSplatThreads, 0, st, rl, rs,
                           lb, vorder.get(), seg_start.get(), seg.get(), in, pre_norm, vals,
                           other);
        return;
    }
    const int Q = value_row(L) / 4;
    float4* rw = reinterpret_cast<float4*>(rows.ensure((size_t)N * Q * 4));
    const int tile = live ? dom_tile : slice_tile_for(L);
    require(tile > 0, DCRF_E_STATE, "splat: live images without prepare_live");
    const size_t psmem = sizeof(float) * kPadWarps * (size_t)((tile * L + 3) & ~3);
    launch_chained(Q == 6 ? pad_rows_kernel<6> : pad_rows_kernel<0>,
                   unit_grid(N, tile * kPadWarps, live, 32 * kPadWarps), 32 * kPadWarps, psmem, st, N, L, Q, tile, in,
                   pre_norm, rw, live_of(kDomTile),
                   live ? (const long*)(dom_base.get() + (long)kDomPix * (images + 1)) : nullptr, (int)aligned16(in));
    const int hb = !concatenated && n_huge <= kHugePerSM * sm_count() ? n_huge : 0;
    const SplatRange rl{hb, n_long - hb, live_of(kDomLong)};
    const int lb = rl.count ? unit_grid(rl.count, kSplatWarps, live, kSplatThreads) : 0;
    const int sb = n_short ? unit_grid((long)n_short * Q, kSplatThreads, live, kSplatThreads) : 0;
    const size_t smem = hb + lb ? (size_t)kSplatWarps * splat_ring_bytes(std::min(Q, 8)) : 0;
    auto kern = Q == 6 ? splat_rows_kernel<6> : splat_rows_kernel<0>;
    if (smem > 48 * 1024)  // opt-in size: a per-device function attribute, set on every such call
        DCRF_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    if (hb + lb + sb)
        launch_chained(kern, hb + lb + sb, kSplatThreads, smem, st, rl, rs, hb, lb, Q, vorder.get(),
                       seg_start.get(), seg.get(), (const float4*)rw,
                       reinterpret_cast<float4*>(vals), reinterpret_cast<float4*>(other));
}

namespace {
constexpr int kTuneMinPixels = 1 << 18;  // smaller lattices keep the default shapes
std::mutex g_tune_mu;
std::vector<std::pair<std::vector<long>, FilterShape>>& tune_cache() {
    static auto* c = new std::vector<std::pair<std::vector<long>, FilterShape>>();  // never destroyed
    return *c;
}
bool autotune_enabled() {
    static const bool on = [] {
        const char* v = std::getenv("DCRF_AUTOTUNE");
        return !(v && v[0] == '0');
    }();
    return on;
}
}  // namespace

void Lattice::tune_shape(int L) {
    shape_L = L;  // also when the defaults stay
    if (N < kTuneMinPixels || !autotune_enabled()) return;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    DCRF_CUDA(cudaStreamIsCapturing(stream, &cs));
    if (cs != cudaStreamCaptureStatusNone) {  // no timing inside a capture: defaults, tuned next time
        shape_L = 0;
        return;
    }
    int dev = 0;
    DCRF_CUDA(cudaGetDevice(&dev));
    int lg = 0;
    while ((1L << (lg + 1)) <= (long)N) lg++;
    const std::vector<long> key = {dev, L, d, lg, M / std::max(N / 64, 1)};
    {
        std::lock_guard<std::mutex> lk(g_tune_mu);
        for (const auto& e : tune_cache())
            if (e.first == key) {
                shape = e.second;
                return;
            }
    }
    const int Lp = value_row(L);
    cudaStream_t st = stream;
    cudaEvent_t e0, e1;
    DCRF_CUDA(cudaEventCreate(&e0));
    DCRF_CUDA(cudaEventCreate(&e1));
    auto timed = [&](auto&& fn) {
        fn();  // warm
        DCRF_CUDA(cudaEventRecord(e0, st));
        for (int r = 0; r < 3; r++) fn();
        DCRF_CUDA(cudaEventRecord(e1, st));
        DCRF_CUDA(cudaEventSynchronize(e1));
        float ms = 0.0f;
        DCRF_CUDA(cudaEventElapsedTime(&ms, e0, e1));
        return ms;
    };
    FilterShape best;
    float* src = va.get();
    float* dst = vb.get();
    float tbest;
    const int Q = Lp / 4;
    const long MQ = (long)M * Q;
    tbest = 1e30f;
    for (int bt : {128, 256, 512}) {
        const float t = timed([&] {
            launch_chained(blur4_kernel<6>, ceil_div(MQ, bt), bt, 0, st, M, Q, nbr.get(), (const float*)src, dst,
                           Live{});
        });
        if (t < tbest) tbest = t, best.blur_threads = bt;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    DCRF_LAUNCH_CHECK();
    shape = best;
    std::lock_guard<std::mutex> lk(g_tune_mu);
    tune_cache().push_back({key, best});
}

void Lattice::splat_blur(const float* in, int L, bool reverse, const float* pre_norm) {
    require(L >= 1, DCRF_E_ARG, "compute: L must be >= 1");
    const int Lp = value_row(L);
    ensure_values((size_t)Lp);
    if (L == 21 && shape_L != L) tune_shape(L);
    cudaStream_t st = stream;
    const long ML = (long)M * L;
    float *src = va.get(), *dst = vb.get();
    // A batched solve's live images: only their lists, vertices and pixels.
    const bool live = live_n != nullptr;
    splat(in, L, pre_norm, src);
    const bool seq = L <= 2;
    const int Q = Lp / 4;
    const long MQ = (long)M * Q;
    const Live lvv = live_of(kDomVert);
    for (int jj = 0; jj <= d; jj++) {
        const int j = reverse ? d - jj : jj;
        const int2* nb = nbr.get() + (long)j * M;
        if (seq) {
            launch_chained(blur_kernel<true>, unit_grid(ML, kTB, live, kTB), kTB, 0, st, M, L, nb, src, dst, lvv);
        } else if (Q == 6) {
            const int bt = shape.blur_threads;
            launch_chained(blur4_kernel<6>, unit_grid(MQ, bt, live, bt), bt, 0, st, M, Q, nb, src, dst, lvv);
        } else {
            launch_chained(blur4_kernel<0>, unit_grid(MQ, kTB, live, kTB), kTB, 0, st, M, Q, nb, src, dst, lvv);
        }
        std::swap(src, dst);
    }
    plain_vals = src;
    plain_L = L;
}

int Lattice::slice_tile_for(int L) const { return slice_tile_max(kSliceTile, d, L); }

void Lattice::slice(float* out, int L, const SliceEpilogue& ep) {
    require(plain_vals && plain_L == L, DCRF_E_STATE, "slice: no splat_blur for this label count before it");
    cudaStream_t st = stream;
    const long NL = (long)N * L;
    const float* src = plain_vals;
    const float alpha = 1.0f / (1.0f + std::pow(2.0f, (float)-d));
    const bool live = live_n != nullptr;
    if (L <= 2) {
        launch_chained(slice_kernel<true, 0, 0>, unit_grid(NL, kTB, live, kTB), kTB, 0, st, N, L, d, offset.get(),
                       bary.get(), src, alpha, out, ep, live_of(kDomPix));
    } else {
        const int Q = value_row(L) / 4;
        // live images: tiles of each image's pixels, the size prepare_live fixed
        const int tile = live ? dom_tile : slice_tile_for(L);
        require(tile > 0, DCRF_E_STATE, "slice: live images without prepare_live");
        const size_t smem = kSliceWarps * slice_warp_bytes(tile, d, L);
        const int vec = aligned16(out) && (!ep.base || aligned16(ep.base));
        const long* pix_base = live ? dom_base.get() + (long)kDomPix * (images + 1) : nullptr;
        auto sl = [&](auto kern) {
            launch_chained(kern, unit_grid(N, tile * kSliceWarps, live, 32 * kSliceWarps), 32 * kSliceWarps, smem, st, N,
                           L, Q, d, tile, offset.get(), bary.get(), reinterpret_cast<const float4*>(src), alpha, out,
                           ep, live_of(kDomTile), pix_base, vec, (const float*)nullptr, (double*)nullptr);
        };
        if (d == 5 && L == 21) sl(slice_rows_kernel<5, 6, 21, false>);
        else if (d == 2 && L == 21) sl(slice_rows_kernel<2, 6, 21, false>);
        else if (d == 5) sl(slice_rows_kernel<5, 0, 0, false>);
        else if (d == 2) sl(slice_rows_kernel<2, 0, 0, false>);
        else sl(slice_rows_kernel<0, 0, 0, false>);
    }
    DCRF_LAUNCH_CHECK();
}

// Warps of slice_dot's grid: 12 blocks per SM fill it, each walking its tiles.
int Lattice::dot_partials() { return sm_count() * 12 * kSliceWarps; }

int Lattice::slice_dot(const float* dot, double* partials, int L, const SliceEpilogue& ep) {
    require(plain_vals && plain_L == L && L > 2 && !ep.base, DCRF_E_STATE, "slice_dot: no splat_blur before it");
    const int Q = value_row(L) / 4, tile = slice_tile_for(L);
    const float alpha = 1.0f / (1.0f + std::pow(2.0f, (float)-d));
    const int grid = std::min(ceil_div(N, tile * kSliceWarps), sm_count() * 12);
    auto sl = [&](auto kern) {
        launch_chained(kern, grid, 32 * kSliceWarps, kSliceWarps * slice_warp_bytes(tile, d, L), stream, N, L, Q, d,
                       tile, offset.get(), bary.get(), reinterpret_cast<const float4*>(plain_vals), alpha,
                       (float*)nullptr, ep, Live{}, (const long*)nullptr, (int)aligned16(dot), dot, partials);
    };
    if (d == 5 && L == 21) sl(slice_rows_kernel<5, 6, 21, true>);
    else if (d == 2 && L == 21) sl(slice_rows_kernel<2, 6, 21, true>);
    else sl(slice_rows_kernel<0, 0, 0, true>);
    DCRF_LAUNCH_CHECK();
    return grid * kSliceWarps;
}

void Lattice::compute_ord(float* out, const float* Q, int L, const SliceEpilogue& ep) {
    require(L >= 1, DCRF_E_ARG, "compute_ord: L must be >= 1");
    const long NL = (long)N * L;
    float2* bins = obins.ensure((size_t)NL);
    ord_bins(bins, Q, NL, stream);
    compute_ord_bins(out, bins, L, ep, nullptr);
}

void rescaled_bins(float2* bins, const float* Q, long n, const float* qminmax, cudaStream_t st) {
    if (aligned16(Q) && aligned16(bins)) {
        const long n4 = n / 4;
        if (n4) launch(rescaled_bins4_kernel, ceil_div(n4, kTB), kTB, 0, st, n4, reinterpret_cast<const float4*>(Q),
                       qminmax, reinterpret_cast<float4*>(bins));
        if (n > 4 * n4)
            launch(rescaled_bins_kernel, 1, kTB, 0, st, n - 4 * n4, Q + 4 * n4, qminmax, bins + 4 * n4);
    } else {
        launch(rescaled_bins_kernel, ceil_div(n, kTB), kTB, 0, st, n, Q, qminmax, bins);
    }
    DCRF_LAUNCH_CHECK();
}

int slice_grid(long n) { return ceil_div(n, kTB); }

void Lattice::compute_ord_bins(float* out, const float2* bins, int L, const SliceEpilogue& ep,
                               const GapFusion* gap) {
    ord_splat_blur(bins, L);
    ord_slice(out, bins, L, ep, gap);
}

void Lattice::ord_splat_blur(const float2* bins, int L) {
    require(L >= 1, DCRF_E_ARG, "compute_ord: L must be >= 1");
    const size_t row = (size_t)L * kOrdW;
    ensure_values(row);
    cudaStream_t st = stream;
    float *src = va.get(), *dst = vb.get();
    // Row 0 is the zero row that absent neighbours read.
    DCRF_CUDA(cudaMemsetAsync(src, 0, sizeof(float) * row, st));
    DCRF_CUDA(cudaMemsetAsync(dst, 0, sizeof(float) * row, st));
    const int n_short = M - n_long;
    if (n_long && L <= kOrdBlockMaxL) {
        // Lists longer than kHugeList (the first n_huge of the order) are
        // shared by blocks of kHugeLabels labels x 10 bins, so that they
        // finish early; the rest take one block per list with the bin split
        // that issues the fewest instructions per entry.
        auto run = [&](int G, int kb, int first, int count, cudaStream_t rs) {
            if (count <= 0) return;
            const int kblocks = (L + kb - 1) / kb;
            const int threads = ((kb * G + 31) / 32) * 32;
            const size_t smem = ord_block_smem(kb);
            auto kern = G == 10 ? ord_splat_block_kernel<10>
                      : G == 5  ? ord_splat_block_kernel<5>
                      : G == 3  ? ord_splat_block_kernel<3>
                      : G == 2  ? ord_splat_block_kernel<2>
                                : ord_splat_block_kernel<1>;
            if (smem > 48 * 1024)  // opt-in size: a per-device function attribute, set on every such call
                DCRF_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            launch(kern, count * kblocks, threads, smem, rs, L, kb, kblocks, vorder.get() + first,
                   seg_start.get(), seg.get(), bins, src);
        };
        // The very long lists set the length of their kernel while leaving
        // most SMs idle; they run on a high-priority side stream, forked
        // after the value buffers are ready and joined before the blur, so
        // the other splats (disjoint vertex rows) fill those SMs meanwhile.
        if (n_huge > 0) {
            ensure_aux();
            DCRF_CUDA(cudaEventRecord(ev_fork, st));
            DCRF_CUDA(cudaStreamWaitEvent(aux, ev_fork, 0));
            run(10, kHugeLabels, 0, n_huge, aux);
            DCRF_CUDA(cudaEventRecord(ev_join, aux));
        }
        run(ord_groups_cheapest(L), L, n_huge, n_long - n_huge, st);
    } else if (n_long) {
        launch(ord_splat_kernel, ceil_div(2L * n_long, kStageWarps), 32 * kStageWarps, 0, st, n_long, L,
               vorder.get(), seg_start.get(), seg.get(), bins, src);
    }
    if (n_short)
        launch(ord_splat_short_kernel<0>, ceil_div((long)n_short * L, kTB), kTB, 0, st, n_short, L,
               vorder.get() + n_long, seg_start.get(), seg.get(), bins, src);
    if (n_long && L <= kOrdBlockMaxL && n_huge > 0) DCRF_CUDA(cudaStreamWaitEvent(st, ev_join, 0));
    const int row4 = (int)(row / 4);
    for (int j = 0; j <= d; j++) {
        auto kern = row4 == 105 ? ord_blur_kernel<105> : ord_blur_kernel<0>;  // 105 = 20 bins x 21 labels / 4
        launch(kern, ceil_div((long)M * row4, kTB), kTB, 0, st, M, row4, nbr.get() + (long)j * M,
               reinterpret_cast<const float4*>(src), reinterpret_cast<float4*>(dst));
        std::swap(src, dst);
    }
    ord_vals = src;
}

void Lattice::ord_slice_pair(float* out, const float2* bins, int L, const Lattice& a, const SliceEpilogue& ea,
                             const Lattice& b, const SliceEpilogue& eb, const GapFusion* gap) {
    require(a.ord_vals && b.ord_vals, DCRF_E_STATE, "ord_slice_pair: no ord_splat_blur before it");
    require(a.N == b.N, DCRF_E_ARG, "ord_slice_pair: lattices over different pixel counts");
    const long NL = (long)a.N * L;
    const OrdSliceTerm t0{a.offset.get(), a.bary.get(), a.ord_vals, a.d, 1.0f / (1.0f + std::pow(2.0f, (float)-a.d)),
                          ea};
    const OrdSliceTerm t1{b.offset.get(), b.bary.get(), b.ord_vals, b.d, 1.0f / (1.0f + std::pow(2.0f, (float)-b.d)),
                          eb};
    const GapFusion gf = gap ? *gap : GapFusion{};
    auto sl = [&](auto kern) {
        launch(kern, ceil_div(NL, kTB), kTB, 0, a.stream, a.N, L, t0, t1, bins, out, gf);
    };
    if (L == 21 && a.d == 2 && b.d == 5) {
        launch(gap ? ord_slice_pair_staged<true> : ord_slice_pair_staged<false>, ceil_div(NL, kTB), kTB, 0,
               a.stream, a.N, t0, t1, bins, out, gf);
    } else if (gap) {
        sl(ord_slice_pair_kernel<true, 0, 0, 0>);
    } else {
        sl(ord_slice_pair_kernel<false, 0, 0, 0>);
    }
    DCRF_LAUNCH_CHECK();
}

void Lattice::ord_slice(float* out, const float2* bins, int L, const SliceEpilogue& ep, const GapFusion* gap) {
    require(ord_vals, DCRF_E_STATE, "ord_slice: no ord_splat_blur before it");
    cudaStream_t st = stream;
    const long NL = (long)N * L;
    const float* src = ord_vals;
    const float alpha = 1.0f / (1.0f + std::pow(2.0f, (float)-d));
    const GapFusion gf = gap ? *gap : GapFusion{};
    auto sl = [&](auto kern) {
        launch(kern, ceil_div(NL, kTB), kTB, 0, st, N, L, d, offset.get(), bary.get(), src, bins, alpha, out, ep, gf);
    };
    if (gap) {
        if (L == 21 && d == 5) sl(ord_slice_kernel<true, 5, 21>);
        else if (L == 21 && d == 2) sl(ord_slice_kernel<true, 2, 21>);
        else sl(ord_slice_kernel<true, 0, 0>);
    } else {
        if (L == 21 && d == 5) sl(ord_slice_kernel<false, 5, 21>);
        else if (L == 21 && d == 2) sl(ord_slice_kernel<false, 2, 21>);
        else sl(ord_slice_kernel<false, 0, 0>);
    }
    DCRF_LAUNCH_CHECK();
}


// ---------------------------------------------------------------------------
// The restricted ordered filter (seqCompute_upper_minus_lower_ord_restricted,
// src/permutohedral.cpp:702-900).
//
// Splat, per (vertex, label) and both passes: the vertex's list in pixel
// order, first the pixels outside pI with their Q values (only in a store
// call; the sums are then kept), then the pixels of pI with their rQ values.
// That is the reference's order per bin: its outside-pI loop runs over all
// pixels before its pI loop.
__global__ void ord_splat_restricted_kernel(int M, int L, const int* __restrict__ seg_start,
                                            const int2* __restrict__ seg,
                                            const int* __restrict__ pos, const float2* __restrict__ ebins,
                                            const float2* __restrict__ rbins, float* __restrict__ stored,
                                            float* __restrict__ vals, unsigned char* __restrict__ active, int store) {
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long)M * L) return;
    const int v = (int)(t / L), k = (int)(t - (long)v * L);
    const int s0 = seg_start[v], s1 = seg_start[v + 1];
    const long rowoff = (long)(v + 1) * kOrdW * L + k;
    unsigned long long acc[kRes];  // (lower, upper) sums of bin b
    if (store) {
#pragma unroll
        for (int b = 0; b < kRes; b++) acc[b] = 0ull;
        bool any = false;
        for (int s = s0; s < s1; s++) {
            const int p = seg[s].x;
            if (pos[p] >= 0) {
                any = true;
                continue;
            }
            const float2 x = ebins[(long)p * L + k];
            const float w = entry_w(seg[s]);
            const unsigned long long w2 = pack2(w, w);
#pragma unroll
            for (int b = 0; b < kRes; b++) ord_step2(acc[b], x.x, x.y, (float)b, w2);
        }
#pragma unroll
        for (int b = 0; b < kRes; b++) {
            const float2 r = unpack2(acc[b]);
            stored[rowoff + (long)b * L] = r.x;
            stored[rowoff + (long)(kRes + b) * L] = r.y;
        }
        if (k == 0) active[v] = any ? 1 : 0;
    } else {
#pragma unroll
        for (int b = 0; b < kRes; b++)
            acc[b] = pack2(stored[rowoff + (long)b * L], stored[rowoff + (long)(kRes + b) * L]);
    }
    for (int s = s0; s < s1; s++) {
        const int ii = pos[seg[s].x];
        if (ii < 0) continue;
        const float2 x = rbins[(long)ii * L + k];
        const float w = entry_w(seg[s]);
        const unsigned long long w2 = pack2(w, w);
#pragma unroll
        for (int b = 0; b < kRes; b++) ord_step2(acc[b], x.x, x.y, (float)b, w2);
    }
#pragma unroll
    for (int b = 0; b < kRes; b++) {
        const float2 r = unpack2(acc[b]);
        vals[rowoff + (long)b * L] = r.x;
        vals[rowoff + (long)(kRes + b) * L] = r.y;
    }
}

// Blur of the active vertices only; the others keep whatever their row of dst
// holds (:773-789: the reference's two buffers swap after every axis, so an
// inactive vertex reads as 0 after odd axes and as its splat after even ones).
__global__ void ord_blur_active_kernel(int M, int row4, const int2* __restrict__ nbr,
                                       const unsigned char* __restrict__ active, const float4* __restrict__ src,
                                       float4* __restrict__ dst) {
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long)M * row4) return;
    const int v = (int)(t / row4), c = (int)(t - (long)v * row4);
    if (!active[v]) return;
    const int2 nb = nbr[v];
    const float4 a = src[(long)(v + 1) * row4 + c];
    const float4 p = src[(long)nb.x * row4 + c];
    const float4 q = src[(long)nb.y * row4 + c];
    float4 r;
    r.x = fadd(a.x, fmul(0.5f, fadd(p.x, q.x)));
    r.y = fadd(a.y, fmul(0.5f, fadd(p.y, q.y)));
    r.z = fadd(a.z, fmul(0.5f, fadd(p.z, q.z)));
    r.w = fadd(a.w, fmul(0.5f, fadd(p.w, q.w)));
    dst[(long)(v + 1) * row4 + c] = r;
}

// Slice at the pI pixels (:791-802, :885-896), as ord_slice_kernel does for
// every pixel; out [nP][L] starts from 0.
__global__ void ord_slice_restricted_kernel(int nP, int L, int d, const int* __restrict__ pI,
                                            const int* __restrict__ offset, const float* __restrict__ bary,
                                            const float* __restrict__ vals, const float2* __restrict__ rbins,
                                            float alpha, float* out, SliceEpilogue ep) {
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long)nP * L) return;
    const int ii = (int)(t / L), k = (int)(t - (long)ii * L);
    const int i = pI[ii], d1 = d + 1;
    const float2 bp = rbins[t];
    const int cl = ord_lower_of(bp), cu = ord_upper_of(bp);
    float acc = 0.0f;
    for (int j = 0; j <= d; j++) {
        const int o = offset[(long)i * d1 + j];
        const float w = bary[(long)i * d1 + j];
        acc = fadd(acc, fmul(vals[((long)(o + 1) * kOrdW + cl) * L + k], fmul(-w, alpha)));
    }
    for (int j = 0; j <= d; j++) {
        const int o = offset[(long)i * d1 + j];
        const float w = bary[(long)i * d1 + j];
        acc = fadd(acc, fmul(vals[((long)(o + 1) * kOrdW + kRes + cu) * L + k], fmul(w, alpha)));
    }
    out[t] = apply_epilogue(acc, t, i, k, ep);
}

__global__ void scatter_pos_kernel(int nP, const int* __restrict__ pI, int* __restrict__ pos) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < nP) pos[pI[t]] = t;
}

void Lattice::compute_ord_restricted(float* rout, const float* rQ, const int* pI, int nP, const float* Q, int L,
                                     bool store, const SliceEpilogue& ep) {
    require(L >= 1, DCRF_E_ARG, "compute_ord_restricted: L must be >= 1");
    require(nP >= 0 && nP <= N, DCRF_E_ARG, "compute_ord_restricted: pI larger than the lattice");
    require(store || r_L == L, DCRF_E_STATE,
            "compute_ord_restricted: no stored splat for this label count (call with store first)");
    require(!store || Q, DCRF_E_ARG, "compute_ord_restricted: store needs Q");
    cudaStream_t st = stream;
    const long row = (long)L * kOrdW, cells = (long)(M + 1) * row;
    float* stored = r_stored.ensure((size_t)cells);
    float* a = r_a.ensure((size_t)cells);
    float* b = r_b.ensure((size_t)cells);
    unsigned char* active = r_active.ensure((size_t)std::max(M, 1));
    int* pos = r_pos.ensure((size_t)N);
    float2* rb = r_bins.ensure((size_t)std::max<long>((long)nP * L, 1));
    launch(fill_int_kernel, ceil_div(N, kTB), kTB, 0, st, (long)N, -1, pos);
    if (nP) {
        launch(scatter_pos_kernel, ceil_div(nP, kTB), kTB, 0, st, nP, pI, pos);
        ord_bins(rb, rQ, (long)nP * L, st);
    }
    const float2* eb = nullptr;
    if (store) {
        float2* e = r_ebins.ensure((size_t)N * L);
        ord_bins(e, Q, (long)N * L, st);
        eb = e;
        r_L = 0;  // until this call has stored its splat
    }
    DCRF_CUDA(cudaMemsetAsync(a, 0, sizeof(float) * row, st));      // row 0: the absent neighbour
    DCRF_CUDA(cudaMemsetAsync(b, 0, sizeof(float) * cells, st));    // new_values_ starts zeroed
    if (M)
        launch(ord_splat_restricted_kernel, ceil_div((long)M * L, kTB), kTB, 0, st, M, L, seg_start.get(),
               seg.get(), (const int*)pos, eb, (const float2*)rb, stored, a, active, (int)store);
    float *src = a, *dst = b;
    const int row4 = (int)(row / 4);
    for (int j = 0; j <= d; j++) {
        if (M)
            launch(ord_blur_active_kernel, ceil_div((long)M * row4, kTB), kTB, 0, st, M, row4,
                   nbr.get() + (long)j * M, (const unsigned char*)active, reinterpret_cast<const float4*>(src),
                   reinterpret_cast<float4*>(dst));
        std::swap(src, dst);
    }
    const float alpha = 1.0f / (1.0f + std::pow(2.0f, (float)-d));
    if (nP)
        launch(ord_slice_restricted_kernel, ceil_div((long)nP * L, kTB), kTB, 0, st, nP, L, d, pI, offset.get(),
               bary.get(), (const float*)src, (const float2*)rb, alpha, rout, ep);
    DCRF_LAUNCH_CHECK();
    if (store) r_L = L;
}

}  // namespace dcrf
