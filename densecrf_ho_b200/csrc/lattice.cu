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

#include "lattice_device.cuh"

namespace dcrf {

namespace {

constexpr int kEmpty = -1;
constexpr int kStageWarps = 2;   // warps (splat lists) per splat block
constexpr int kStages = 3;       // shared-memory ring depth, in chunks
constexpr int kChunk = 32;       // entries per chunk (13 KB of ring per warp: 16 warps / SM)

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

// K1: one thread per (padded) pixel.  DC: d as a compile-time constant, so that
// every per-pixel array lives in registers (with run-time indexes they were in
// local memory: 56 us for 640x480, d = 5), or 0 (d <= DM).
struct ElevateScale {
    float s[16];  // scale_factor_ per coordinate
};
template <int DM, int DC>
__global__ void elevate_kernel(const float* __restrict__ feat, int N, int Np, int drt, ElevateScale scale,
                               int4* __restrict__ ekeys, int* __restrict__ rank_out, float* __restrict__ bary_out) {
    constexpr int KW = (DM + 7) / 8;
    constexpr int U = DC ? DC : DM;  // loop bounds; run-time d stops earlier
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= Np) return;
    const int d = DC ? DC : drt;
    const int d1 = d + 1;
    const float invdp1 = 1.0f / (float)d1, dp1 = (float)d1;
    float f[U], el[U + 1], rem0[U + 1], rk[U + 1], b[U + 2];
#pragma unroll
    for (int j = 0; j < U; j++)
        if (j < d) f[j] = k < N ? feat[(long)k * d + j] : 0.0f;
    // Elevation (:213-219): sm accumulates from the last coordinate down.
    float sm = 0.0f;
#pragma unroll
    for (int j = U; j > 0; j--)
        if (j <= d) {
            const float cf = fmul(f[j - 1], scale.s[j - 1]);
            el[j] = fsub(sm, fmul((float)j, cf));
            sm = fadd(sm, cf);
        }
    el[0] = sm;
    // Closest 0-coloured simplex (:222-232).
    float sum = 0.0f;
#pragma unroll
    for (int i = 0; i <= U; i++)
        if (i <= d) {
            const float v = cvt_rne(fmul(invdp1, el[i]));
            rem0[i] = fmul(v, dp1);
            sum = fadd(sum, v);
        }
    // Rank (:235-245).
#pragma unroll
    for (int i = 0; i <= U; i++) rk[i] = 0.0f;
#pragma unroll
    for (int i = 0; i < U; i++)
        if (i < d) {
            const float di = fsub(el[i], rem0[i]);
#pragma unroll
            for (int j = i + 1; j <= U; j++)
                if (j <= d) {
                    const float dj = fsub(el[j], rem0[j]);
                    const float c = (di < dj) ? 1.0f : 0.0f;
                    rk[i] = fadd(rk[i], c);
                    rk[j] = fadd(rk[j], fsub(1.0f, c));
                }
        }
    // Back onto the plane (:248-254).
#pragma unroll
    for (int i = 0; i <= U; i++)
        if (i <= d) {
            rk[i] = fadd(rk[i], sum);
            const float add = rk[i] < 0.0f ? dp1 : 0.0f;
            const float sub = rk[i] >= dp1 ? dp1 : 0.0f;
            const float t = fsub(add, sub);
            rk[i] = fadd(rk[i], t);
            rem0[i] = fadd(rem0[i], t);
        }
    // Barycentric coordinates (:257-275).
#pragma unroll
    for (int i = 0; i < U + 2; i++) b[i] = 0.0f;
#pragma unroll
    for (int i = 0; i <= U; i++)
        if (i <= d) {
            const float v = fmul(fsub(el[i], rem0[i]), invdp1);
            int p = (int)fsub((float)d, rk[i]);
            p = min(max(p, 0), d);  // in range for finite features; guards NaN input
#pragma unroll
            for (int q = 0; q < U + 2; q++) {
                if (q == p) b[q] = fadd(b[q], v);
                if (q == p + 1) b[q] = fsub(b[q], v);
            }
        }
    float last = 0.0f;  // b[d + 1]
#pragma unroll
    for (int q = 0; q < U + 2; q++)
        if (q == d1) last = b[q];
    b[0] = fadd(b[0], fadd(1.0f, last));
    // Keys of the d+1 vertices (:280-287); canonical simplex (:183-188).
#pragma unroll
    for (int r = 0; r <= U; r++) {
        if (r > d) break;
        Key<KW> key;
        key_zero(key);
#pragma unroll
        for (int i = 0; i < U; i++)
            if (i < d) {
                const int ri = (int)rk[i];
                const int canon = (ri <= d - r) ? r : r - d1;
                key_set(key, i, (int16_t)(int)fadd(rem0[i], (float)canon));
            }
        const long e = (long)k * d1 + r;
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
            // the slot only ever gets smaller: once it is at most e, e has no part in it
            if (cur > e) atomicMin(table + h, e);
            entry_slot[e] = (int)h;
            return;
        }
        h = (h + 1) & mask;
    }
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

// K5: the splat lists from the entries sorted by vertex: (pixel, weight) pairs,
// and every list's start where the vertex changes (vertices without entries --
// those only padding pixels touch -- start where the next list does).
__global__ void seg_fill_kernel(int E, int M, int d1, const int* __restrict__ sorted_vertices,
                                const int* __restrict__ sorted_entries, const float* __restrict__ bary,
                                int2* __restrict__ seg, int* __restrict__ seg_start) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s > E) return;
    const int v = s < E ? sorted_vertices[s] : M, before = s > 0 ? sorted_vertices[s - 1] : -1;
    for (int u = before + 1; u <= v; u++) seg_start[u] = s;
    if (s < E) {
        const int e = sorted_entries[s];
        seg[s] = make_int2(e / d1, __float_as_int(bary[e]));
    }
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

// The lists a splat launch covers: positions [first, first + count) of
// `order`, or the live images' positions of the domain behind lv.
struct SplatRange {
    int first = 0, count = 0;
    Live lv;
};
__device__ __forceinline__ int splat_vertex(const SplatRange& r, const int* __restrict__ order, long u) {
    return order[r.lv.n ? live_unit(r.lv, u) : r.first + u];
}

// Streams the list [s0, s1) of one vertex through the per-warp ring:
// ring[slot][e] holds this chunk's entries' values, mw[slot] their weights and,
// with a norm, mn[slot] their factors; consume(slot, n) is called once per
// chunk, in order.
template <typename Consume>
__device__ __forceinline__ void stream_list(int s0, int s1, int L, int k, bool act, int lane,
                                            const int2* __restrict__ seg, const float* __restrict__ src,
                                            const float* __restrict__ norm, float (*ring)[kChunk][32],
                                            float (*mw)[kChunk], float (*mn)[kChunk], Consume&& consume) {
    const int nch = (s1 - s0 + kChunk - 1) / kChunk;
    auto pix_of = [&](int c) {
        const int base = s0 + c * kChunk;
        return (c < nch && lane < s1 - base) ? seg[base + lane].x : 0;
    };
    auto issue = [&](int c, int pc) {
        const int slot = c % kStages, base = s0 + c * kChunk, n = min(kChunk, s1 - base);
        if (lane < n) cp_async4(&mw[slot][lane], &seg[base + lane].y);
        if (norm && lane < n) cp_async4(&mn[slot][lane], norm + pc);
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

// The splat of input rows as they are, for the allocation-free filter and where
// memory is short: neither holds the padded copy of the splat below.  The long
// lists, one warp per vertex; rows of Lp values, those past L zero.  PLAIN: no
// norm, no live images and rows of L values (the allocation-free filter, 640x480,
// two features, 100 labels: 402 us so, 424 with those at run time).
template <bool PLAIN>
__global__ void __launch_bounds__(32 * kStageWarps)
    splat_kernel(SplatRange r, int L, int Lp, const int* __restrict__ order, const int* __restrict__ seg_start,
                 const int2* __restrict__ seg, const float* __restrict__ in, const float* __restrict__ norm_,
                 float* __restrict__ vals) {
    const float* norm = PLAIN ? nullptr : norm_;
    if (PLAIN) {
        Lp = L;
        r.lv = Live{};
    }
    __shared__ float ring[kStageWarps][kStages][kChunk][32];
    __shared__ float mw[kStageWarps][kStages][kChunk], mn[kStageWarps][kStages][kChunk];
    const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long total = live_total(r.lv, r.count);
    for (long unit = (long)blockIdx.x * kStageWarps + wib; unit < total; unit += (long)gridDim.x * kStageWarps) {
        const int v = splat_vertex(r, order, unit);  // warp-uniform
        const int s0 = seg_start[v], s1 = seg_start[v + 1];
        for (int kb = 0; kb < L; kb += 32) {
            const int k = kb + lane;
            const bool act = k < L;
            float acc = 0.0f;
            stream_list(s0, s1, L, k, act, lane, seg, in, norm, ring[wib], mw[wib], mn[wib], [&](int slot, int n) {
#pragma unroll 4
                for (int e = 0; e < n; e++) {
                    const float x = ring[wib][slot][e][lane];
                    acc = fadd(acc, fmul(mw[wib][slot][e], norm ? fmul(x, mn[wib][slot][e]) : x));
                }
            });
            if (k < Lp) vals[(long)(v + 1) * Lp + k] = act ? acc : 0.0f;
        }
    }
}

// ... and the short ones: one thread per (vertex, label).  Also row 0 of both
// value buffers, which absent neighbours read.
template <bool PLAIN>
__global__ void splat_short_kernel(SplatRange r, int L, int Lp, const int* __restrict__ order,
                                   const int* __restrict__ seg_start, const int2* __restrict__ seg,
                                   const float* __restrict__ in, const float* __restrict__ norm_,
                                   float* __restrict__ vals, float* __restrict__ other) {
    const float* norm = PLAIN ? nullptr : norm_;
    if (PLAIN) {
        Lp = L;
        r.lv = Live{};
    }
    const long t0 = (long)blockIdx.x * blockDim.x + threadIdx.x, nt = (long)gridDim.x * blockDim.x;
    for (long t = t0; t < Lp; t += nt) vals[t] = other[t] = 0.0f;
    const long total = live_total(r.lv, r.count) * Lp;
    for (long t = t0; t < total; t += nt) {
        const long u = t / Lp;
        const int k = (int)(t - u * Lp);
        const int v = splat_vertex(r, order, u);
        const int s0 = seg_start[v], s1 = k < L ? seg_start[v + 1] : s0;
        float acc = 0.0f;
#pragma unroll 4
        for (int s = s0; s < s1; s++) {
            const int2 e = seg[s];
            const float x = in[(long)e.x * L + k];
            acc = fadd(acc, fmul(entry_w(e), norm ? fmul(x, norm[e.x]) : x));
        }
        vals[(long)(v + 1) * Lp + k] = acc;
    }
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

// The same where a pixel's row does not fit a warp's tile (row_tiles): a thread
// per 16-byte group, blockIdx.y walking the pixels.  The whole filter at the
// line, 64x48 and five features: 437 us with 3056 labels by tiles, 423 with
// 3057 by these.
__global__ void __launch_bounds__(kTB)
    pad_wide_kernel(int N, int L, int Q, const float* __restrict__ in, float4* __restrict__ rows) {
    const int q = blockIdx.x * kTB + threadIdx.x, n = L - 4 * q;
    grid_release();
    grid_wait();
    if (q >= Q) return;
    for (long i = blockIdx.y; i < N; i += gridDim.y) {
        const float* x = in + i * L + 4 * q;
        rows[i * Q + q] = make_float4(x[0], n > 1 ? x[1] : 0.0f, n > 2 ? x[2] : 0.0f, n > 3 ? x[3] : 0.0f);
    }
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

// The splat for L = 1, 2 (seqCompute; also every normalisation factor; `in`
// null: ones): the
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
                        x[i][k] = in ? in[(long)p[i] * L + k] : 1.0f;
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
                    float x = in ? in[(long)p * L + k] : 1.0f;
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

// Class of a splat list by its length: 0 long, 1 short.
__device__ __forceinline__ int list_class(int c) { return c > kLongList ? 0 : 1; }

// Concatenated lattices: the key (class, image) of each position of the
// length-sorted visiting order, for a second stable sort that groups each
// class's lists by image (longest first within an image), and the number of
// lists per (class, image).
__global__ void class_image_key_kernel(int M, const int* __restrict__ order, const int* __restrict__ seg_start,
                                       const int* __restrict__ vimg, int images, int* __restrict__ keys,
                                       int* __restrict__ per_class_image) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= M) return;
    const int v = order[p];
    const int key = list_class(seg_start[v + 1] - seg_start[v]) * images + vimg[v];
    keys[p] = key;
    atomicAdd(&per_class_image[key], 1);
}

// Sort key of the splat visiting order (stable radix sort ascending): the
// long lists first, longest first, so that their chains start early; the
// short lists after them in vertex-id order.  Ids follow the pixels' scan
// order (first occurrence), so consecutive short lists gather rows of nearby
// pixels and each input row is fetched from DRAM about once although d + 1
// lists read it (sorting the short lists by length too scattered them over
// the whole image).  Lengths count to a sixteenth of a power of two, which
// keeps the classes apart (64 and 1024 are powers of two) and the key in one
// 8-bit radix pass; three passes over exact lengths took 15 launches.  Also
// counts the lists over kLongList and kHugeList entries (n[0], n[1]).
constexpr int kOrderBits = 8;
__global__ void order_key_kernel(int M, const int* __restrict__ seg_start, int* __restrict__ keys,
                                 int* __restrict__ n) {
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    const int c = v < M ? seg_start[v + 1] - seg_start[v] : 0;
    if (v < M) {
        int key = 255;
        if (c > kLongList) {
            const int x = c - 1, e = 31 - __clz(x);  // x >= 64
            key = 254 - min((e - 6) * 16 + ((x >> (e - 4)) & 15), 254);
        }
        keys[v] = key;
    }
    const unsigned l = __ballot_sync(0xffffffffu, c > kLongList), h = __ballot_sync(0xffffffffu, c > kHugeList);
    if ((threadIdx.x & 31) == 0) {
        if (l) atomicAdd(n, __popc(l));
        if (h) atomicAdd(n + 1, __popc(h));
    }
}

// One blur pass along one lattice axis: new = old + 1/2 (n1 + n2).  seqCompute
// evaluates it in double (0.5 is a double literal there, :518).
template <bool SEQ>
__global__ void blur_kernel(int M, int L, const int2* __restrict__ nbr,
                            const float* __restrict__ src, float* __restrict__ dst, Live lv) {
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

// Slice: out(i, k) = sum_j (bary_ij * alpha) * value(o_ij, k) (sseCompute,
// :1046-1051) or sum_j (bary_ij * value) * alpha (seqCompute, :529-534).
template <bool SEQ>
__global__ void slice_kernel(int N, int L, int d, const int* __restrict__ offset,
                             const float* __restrict__ bary, const float* __restrict__ vals,
                             float alpha, float* out, SliceEpilogue ep, Live lv) {
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
// A row's first group (row times Q) is staged as an unsigned product: two value
// buffers of more than 2^32 groups (64 GiB, in blocks of 96) do not fit the
// device, and a 64-bit multiplication at the gather costs (the whole filter,
// 320x240, three features, 12 labels: 80 us staged, 86 multiplied).
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
            s_ow[e] = make_int2((int)((unsigned)(offset[p0 * d1 + e] + 1) * Qn),
                                __float_as_int(fmul(bary[p0 * d1 + e], alpha)));
        if (use_norm)
            for (int e = lane; e < np; e += 32) s_nrm[e] = ep.norm[p0 + e];
        cp_async_wait<0>();
        __syncwarp();
        auto item = [&](int pl, int q) {
            const int2* ow = s_ow + pl * d1;
            const float4* vq = vals + q;
            unsigned long long a0 = 0ull, a1 = 0ull;
            auto add = [&](int2 e) {
                const long row = (long)(unsigned)e.x;
                const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(vq + row);
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

// The slice of rows that do not fit a warp's tile (row_tiles), split as
// pad_wide_kernel: the same sums, no epilogue.
__global__ void __launch_bounds__(kTB)
    slice_wide_kernel(int N, int L, int Q, int d1, const int* __restrict__ offset, const float* __restrict__ bary,
                      const float4* __restrict__ vals, float alpha, float* __restrict__ out) {
    const int q = blockIdx.x * kTB + threadIdx.x, n = L - 4 * q;
    grid_release();
    grid_wait();
    if (q >= Q) return;
    for (long i = blockIdx.y; i < N; i += gridDim.y) {
        unsigned long long a0 = 0ull, a1 = 0ull;
        for (int j = 0; j < d1; j++) {
            const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(vals + (long)(offset[i * d1 + j] + 1) * Q + q);
            const float wa = fmul(bary[i * d1 + j], alpha);
            a0 = add_mul2(a0, wa, v.x);
            a1 = add_mul2(a1, wa, v.y);
        }
        const float2 lo = unpack2(a0), hi = unpack2(a1);
        float* o = out + i * L + 4 * q;
        o[0] = lo.x;
        if (n > 1) o[1] = lo.y;
        if (n > 2) o[2] = hi.x;
        if (n > 3) o[3] = hi.y;
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
    ElevateScale scale{};
    const float inv_std_dev = (float)(std::sqrt(2.0 / 3.0) * (d + 1));
    for (int i = 0; i < d; i++) scale.s[i] = (float)(1.0 / std::sqrt((double)((i + 2) * (i + 1))) * inv_std_dev);

    int4* ekeys = L.ekeys.ensure((size_t)E * KW);
    int* rank = L.rank.ensure(Ereal);
    float* bary = L.bary.ensure(Ereal);
    unsigned cap = 1;
    while ((long)cap < 2 * E) cap <<= 1;
    int* table = L.table.ensure(cap);
    DCRF_CUDA(cudaMemsetAsync(table, 0xff, sizeof(int) * cap, st));
    launch(d == DM ? elevate_kernel<DM, DM> : elevate_kernel<DM, 0>, ceil_div(Np, 128), 128, 0, st, d_features, N, Np,
           d, scale, ekeys, rank, bary);
    int* eslot = L.entry_slot.ensure(E);
    launch(insert_kernel<KW>, ceil_div(E, kTB), kTB, 0, st, ekeys, (int)E, table, cap - 1, eslot);
    int* flags = L.flags.ensure(E);
    int* dtotal = L.total.ensure(4);
    first_flags_scan(eslot, table, (int)E, flags, dtotal, L.scan, st);
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

    // Splat lists: stable sort of the entries by vertex, then the lists' starts.
    int* seg_start = L.seg_start.ensure((size_t)M + 1);
    const int *sorted_v, *sorted_e;
    radix_sort_index(offset, (int)Ereal, bits_for(M), L.sort_keys.ensure(Ereal), L.sort_vals.ensure(Ereal), &sorted_v,
                     &sorted_e, L.sort, st);
    int2* seg = L.seg.ensure(Ereal + kSegPad);
    launch(seg_fill_kernel, ceil_div(Ereal + 1, kTB), kTB, 0, st, (int)Ereal, M, d1, sorted_v, sorted_e,
           (const float*)bary, seg, seg_start);
    int nl[2];
    L.visiting_order(nl);
    L.n_long = nl[0];
    L.n_huge = nl[1];
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

// ROWS: the values lie in rows of Lp / 4 float4 (L > 2) and four labels come
// at a time, else one.  Bound by its gathers' loads, two rows per simplex
// vertex and pixel: 105 -> 57 us at 640x480, five features, 21 labels, by
// taking 16 bytes a load instead of four.
template <int DM, bool ROWS>
__global__ void grad_slice_kernel(int N, int L, int Lp, int d, const int* __restrict__ offset, const int* __restrict__ rank,
                                  const float* __restrict__ vals, const float* __restrict__ x, float alpha,
                                  GradScale sf, float* __restrict__ df) {
    constexpr int G = ROWS ? 4 : 1;  // labels at a time
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
    for (int k0 = 0; k0 < L; k0 += G) {
        float ra[DM + 1][G];
#pragma unroll
        for (int j = 0; j <= DM; j++)
            if (j <= d) {
                float v0[G], v1[G];
                if constexpr (ROWS) {
                    const float4 p = *reinterpret_cast<const float4*>(vals + (long)o0[j] * Lp + k0);
                    const float4 q = *reinterpret_cast<const float4*>(vals + (long)o1[j] * Lp + k0);
                    v0[0] = p.x, v0[1] = p.y, v0[2] = p.z, v0[3] = p.w;
                    v1[0] = q.x, v1[1] = q.y, v1[2] = q.z, v1[3] = q.w;
                } else {
                    v0[0] = vals[(long)o0[j] * Lp + k0];
                    v1[0] = vals[(long)o1[j] * Lp + k0];
                }
#pragma unroll
                for (int c = 0; c < G; c++) ra[j][c] = fsub(fadd(0.0f, fmul(alpha, v0[c])), fmul(alpha, v1[c]));
            }
        float xk[G];
#pragma unroll
        for (int c = 0; c < G; c++) xk[c] = k0 + c < L ? x[(long)i * L + k0 + c] : 0.0f;
#pragma unroll
        for (int c = 0; c < G; c++) {
            if (k0 + c >= L) break;  // a row's padding
            float sm = ra[0][c];
#pragma unroll
            for (int j = 1; j <= DM; j++)
                if (j <= d) {
                    const float v = fmul(sf.s[j - 1], fsub(sm, fmul((float)j, ra[j][c])));
                    grad[j - 1] = fadd(grad[j - 1], fmul(xk[c], v));
                    sm = fadd(sm, ra[j][c]);
                }
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
        launch(L > 2 ? grad_slice_kernel<DM, true> : grad_slice_kernel<DM, false>, ceil_div(N, 128), 128, 0, st, N, L, Lp,
               d, lat.offset.get(), lat.rank.get(), src, dir ? a : b, alpha, sf, df);
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

}  // namespace

// vorder from seg_start (see order_key_kernel); nl: the lists over kLongList and
// kHugeList entries.  Waits for the stream.
void Lattice::visiting_order(int (&nl)[2]) {
    int* dl = total.ensure(4);
    DCRF_CUDA(cudaMemsetAsync(dl, 0, 2 * sizeof(int), stream));
    int* ok = vorder_keys.ensure(std::max(M, 1));
    int* vo = vorder.ensure(std::max(M, 1));
    launch(order_key_kernel, ceil_div(M, kTB), kTB, 0, stream, M, (const int*)seg_start.get(), ok, dl);
    const int *sk, *sv;
    radix_sort_index(ok, M, kOrderBits, ok, vo, &sk, &sv, sort, stream);
    if (sv != vo) DCRF_CUDA(cudaMemcpyAsync(vo, sv, sizeof(int) * M, cudaMemcpyDeviceToDevice, stream));
    DCRF_CUDA(cudaMemcpyAsync(nl, dl, 2 * sizeof(int), cudaMemcpyDeviceToHost, stream));
    DCRF_CUDA(cudaStreamSynchronize(stream));
}

void Lattice::concat_parts(const std::vector<const Lattice*>& parts) {
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
    int nl[2];
    visiting_order(nl);
    int* vo = vorder.get();
    int* ok = vorder_keys.get();
    // Then, stably, by (class, image): each class (long, short lists) holds
    // its lists image by image, longest first within an image, so
    // that an image's lists of a class are one contiguous range of the order
    // (the live-image domains of a batched solve).
    const int B = (int)parts.size();
    DevBuf<int> pci;
    int* per_ci = pci.ensure((size_t)2 * B);
    DCRF_CUDA(cudaMemsetAsync(per_ci, 0, sizeof(int) * 2 * B, st));
    launch(class_image_key_kernel, ceil_div(M, kTB), kTB, 0, st, M, (const int*)vo, (const int*)ss,
           (const int*)vi, B, ok, per_ci);
    int kbits = 1;
    while ((1L << kbits) < 2L * B) kbits++;
    radix_sort_pairs(ok, vo, M, kbits, sort, st);
    DCRF_LAUNCH_CHECK();
    std::vector<int> hci((size_t)2 * B);
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
    build_in([&] {
        N = N_;
        d = d_;
        if (d <= 2) build_impl<2>(*this, d_features);
        else if (d <= 5) build_impl<5>(*this, d_features);
        else if (d <= 8) build_impl<8>(*this, d_features);
        else build_impl<16>(*this, d_features);
    });
}

void Lattice::concat(const std::vector<const Lattice*>& parts) {
    build_in([&] { concat_parts(parts); });
}

template <typename F>
void Lattice::build_in(F&& build) {
    forget();
    for (bool again = false;; again = true) {
        try {
            build();
            return;
        } catch (const Error& e) {
            forget();
            if (again || e.code != DCRF_E_NOMEM ||
                !(give_back() | give_back_quads() | (give_back_others && give_back_others())))
                throw;
            cudaGetLastError();
        } catch (...) {
            forget();
            throw;
        }
    }
}

static bool release_all() { return false; }
template <typename T, typename... Rest>
static bool release_all(DevBuf<T>& b, Rest&... rest) {
    const bool had = b.get() != nullptr;
    b.release();
    return release_all(rest...) | had;
}

bool Lattice::give_back() {
    return release_all(rows, ekeys, table, entry_slot, flags, slot_vid, sort_keys, sort_vals, vorder_keys, scan.block_sums,
                       sort.keys_alt, sort.vals_alt, sort.hist, sort.scan.block_sums);
}

// The ordered filter's buffers beside the value buffers.
bool Lattice::give_back_quads() {
    ord_vals = nullptr;
    ord_T_ready = false;
    return release_all(obins, ord_a, ord_b, ord_plane, ord_T);
}

// No lattice: N = 0 until one is built, and nothing that was computed on the
// former one is taken for this one's.
void Lattice::forget() {
    N = M = 0;
    plain_vals = ord_vals = nullptr;
    plain_L = r_L = 0;
    ord_T_ready = false;
}

void Lattice::ensure_values(size_t row_width) {
    const size_t need = (size_t)(M + 1) * row_width;
    own(va, need);
    own(vb, need);
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
    // The array keeps the previous call's contents: the splat clears the zero
    // rows that absent neighbours read; every other row read below is written
    // first.
    const long ML = (long)M * L, NL = (long)N * L;
    splat_plain(in, L, L, nullptr, src, dst);
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
        launch(slice_kernel<true>, ceil_div(NL, kTB), kTB, 0, st, N, L, d, offset.get(), bary.get(), src, alpha,
               out, ep, Live{});
    else
        launch(slice_kernel<false>, ceil_div(NL, kTB), kTB, 0, st, N, L, d, offset.get(), bary.get(), src, alpha,
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
// Whether four warps' tiles of one pixel fit a block's 48 KB: up to some 3050
// labels.  Only a lattice's own calls can have more (a model's limit is 64).
static bool row_tiles(int d, int L) { return kSliceWarps * slice_warp_bytes(1, d, L) <= (48 << 10); }
static dim3 wide_grid(int N, int Q) { return dim3(ceil_div(Q, kTB), std::min(N, 65535)); }

// The splat without the padded rows, into rows of Lp floats.
void Lattice::splat_plain(const float* in, int L, int Lp, const float* pre_norm, float* vals, float* other) {
    const bool live = live_n != nullptr, plain = !live && !pre_norm && Lp == L;
    const int n_short = M - n_long;
    if (n_long)
        launch(plain ? splat_kernel<true> : splat_kernel<false>, unit_grid(n_long, kStageWarps, live, 32 * kStageWarps),
               32 * kStageWarps, 0, stream, SplatRange{0, n_long, live_of(kDomLong)}, L, Lp, vorder.get(),
               seg_start.get(), seg.get(), in, pre_norm, vals);
    launch(plain ? splat_short_kernel<true> : splat_short_kernel<false>,
           unit_grid((long)n_short * Lp, kTB, live, kTB), kTB, 0, stream,
           SplatRange{n_long, n_short, live_of(kDomShort)}, L, Lp, vorder.get(), seg_start.get(), seg.get(), in,
           pre_norm, vals, other);
}

// The padded rows, or null where there is no memory for them.  Not asked for
// inside a capture, which must not wait for the device.
float* Lattice::rows_or_null(size_t floats) {
    if (rows.n >= floats) return rows.get();
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    DCRF_CUDA(cudaStreamIsCapturing(stream, &cs));
    if (cs != cudaStreamCaptureStatusNone) return nullptr;
    try {
        return rows.ensure(floats);
    } catch (const Error& e) {
        if (e.code != DCRF_E_NOMEM) throw;
        cudaGetLastError();
        return nullptr;
    }
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
    float4* rw = reinterpret_cast<float4*>(rows_or_null((size_t)N * Q * 4));
    if (!rw) {
        splat_plain(in, L, 4 * Q, pre_norm, vals, other);
        return;
    }
    const int tile = live ? dom_tile : slice_tile_for(L);
    require(tile > 0, DCRF_E_STATE, "splat: live images without prepare_live");
    if (!row_tiles(d, L)) {
        require(!live && !pre_norm, DCRF_E_ARG, "splat: too many labels");
        launch_chained(pad_wide_kernel, wide_grid(N, Q), kTB, 0, st, N, L, Q, in, rw);
    } else {
        const size_t psmem = sizeof(float) * kPadWarps * (size_t)((tile * L + 3) & ~3);
        launch_chained(Q == 6 ? pad_rows_kernel<6> : pad_rows_kernel<0>,
                       unit_grid(N, tile * kPadWarps, live, 32 * kPadWarps), 32 * kPadWarps, psmem, st, N, L, Q, tile,
                       in, pre_norm, rw, live_of(kDomTile),
                       live ? (const long*)(dom_base.get() + (long)kDomPix * (images + 1)) : nullptr,
                       (int)aligned16(in));
    }
    const int hb = !concatenated && n_huge <= kHugePerSM * sm_count() ? n_huge : 0;
    const SplatRange rl{hb, n_long - hb, live_of(kDomLong)};
    const int lb = rl.count ? unit_grid(rl.count, kSplatWarps, live, kSplatThreads) : 0;
    const int sb = n_short ? unit_grid((long)n_short * Q, kSplatThreads, live, kSplatThreads) : 0;
    const size_t smem = hb + lb ? (size_t)kSplatWarps * splat_ring_bytes(std::min(Q, 8)) : 0;
    auto kern = Q == 6 ? splat_rows_kernel<6> : splat_rows_kernel<0>;
    // The opt-in is an attribute of the kernel that all threads share: always the
    // largest size there is (eight groups a row).
    if (smem > 48 * 1024)
        DCRF_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       kSplatWarps * splat_ring_bytes(8)));
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

// ord_T: row 0 the weights' sums per vertex in entry order, row j + 1 row j
// blurred along axis j (each row M + 1 floats, the first zero).
void Lattice::ensure_ord_totals() {
    if (ord_T_ready) return;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    DCRF_CUDA(cudaStreamIsCapturing(stream, &cs));
    const long rowT = M + 1;
    float* T = own(ord_T, (size_t)(d + 2) * rowT);
    DCRF_CUDA(cudaMemsetAsync(T, 0, sizeof(float) * (d + 2) * rowT, stream));
    const int n_short = M - n_long;
    const SplatRange rl{0, n_long, Live{}}, rs{n_long, n_short, Live{}};
    const int lb = ceil_div(n_long, kSplatWarps), sb = ceil_div(n_short, kSplatThreads);
    launch_chained(splat_thin_kernel<1>, lb + sb, kSplatThreads, 0, stream, rl, rs, lb, vorder.get(), seg_start.get(),
                   seg.get(), (const float*)nullptr, (const float*)nullptr, T, T + rowT);
    for (int j = 0; j <= d; j++)
        launch_chained(blur_kernel<false>, ceil_div(M, kTB), kTB, 0, stream, M, 1, nbr.get() + (long)j * M,
                       T + j * rowT, T + (j + 1) * rowT, Live{});
    DCRF_LAUNCH_CHECK();
    ord_T_ready = cs == cudaStreamCaptureStatusNone;  // a captured launch has not run yet
}

void Lattice::splat_blur(const float* in, int L, bool reverse, const float* pre_norm) {
    require(L >= 1, DCRF_E_ARG, "compute: L must be >= 1");
    const int Lp = value_row(L);
    // slice_rows_kernel's row index; ensure_values would find no memory either
    require((long)(M + 1) * (Lp / 4) < 1L << 32, DCRF_E_NOMEM, "compute: value buffers over 64 GiB");
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
        launch_chained(slice_kernel<true>, unit_grid(NL, kTB, live, kTB), kTB, 0, st, N, L, d, offset.get(),
                       bary.get(), src, alpha, out, ep, live_of(kDomPix));
    } else if (!row_tiles(d, L)) {
        require(!live && !ep.potts && !ep.base && !ep.zero_base, DCRF_E_ARG, "slice: too many labels");
        const int Q = value_row(L) / 4;
        launch_chained(slice_wide_kernel, wide_grid(N, Q), kTB, 0, st, N, L, Q, d + 1, offset.get(), bary.get(),
                       reinterpret_cast<const float4*>(src), alpha, out);
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
        const bool l21 = L == 21;
        if (d == 5 && l21) sl(slice_rows_kernel<5, 6, 21, false>);
        else if (d == 2 && l21) sl(slice_rows_kernel<2, 6, 21, false>);
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
    const bool l21 = L == 21;
    if (d == 5 && l21) sl(slice_rows_kernel<5, 6, 21, true>);
    else if (d == 2 && l21) sl(slice_rows_kernel<2, 6, 21, true>);
    else sl(slice_rows_kernel<0, 0, 0, true>);
    DCRF_LAUNCH_CHECK();
    return grid * kSliceWarps;
}

}  // namespace dcrf
