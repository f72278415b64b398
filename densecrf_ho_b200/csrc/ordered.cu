// The 10-bin ordered filter (seqCompute_upper_minus_lower_ord,
// src/permutohedral.cpp:548-701) on sm_100a, and its restricted form.
//
// A (vertex, label) holds 20 sums: lower bins lo[0..9] add the weights of the
// entries whose lower bin reaches them (c_lower >= b), upper bins up[0..9]
// those with c_upper <= b, each in entry order.  Two facts keep most of that
// from being computed, stored or moved, with every value bit for bit the
// reference's:
//   - lo[0] and up[9] take every entry, whatever the label: both are T(v), the
//     sum of the vertex's weights, which depends on the lattice alone
//     (Lattice::ord_T keeps it, and its blurred forms, per lattice);
//   - where no entry of a (vertex, label) has a lower bin above b, lo[b+1] is
//     exactly 0 and up[b] is exactly T(v) -- the same chain of adds -- and a
//     blur of such values gives such values again.
// So the 18 other sums are kept as nine pairs (lo[b+1], up[b]), b = 0..8, two
// pairs to a 16-byte quad, five quads per label, and a quad is stored only
// when some entry reaches it; a bit mask per vertex says which are (bit 5 k + q
// for label k's quad q).  A solver's iterates put 94 % of all (pixel, label)
// values in one bin, so on its lattices the lists touch 6 to 40 % of the quads
// (640x480 LP, both lattices); a mask costs 16 bytes per vertex at L = 21.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "lattice_device.cuh"

namespace dcrf {

namespace {

// Programmatic dependent launches (launch_chained) pay while the filter's
// kernels are short (64x48: 59 -> 47 us a call, 320x240 with 5 labels 105 ->
// 91), and cost on long ones, whose successors' early blocks crowd them
// (320x240 with 12 labels 67 -> 74 us, with 40 labels 228 -> 247, 640x480 269
// -> 304; 393 -> 622 where the bins are spread): chained up to 2^19 (pixel,
// label) values.
template <typename... KArgs, typename... Args>
void launch_ord(long values, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                Args&&... args) {
    if (values <= 1L << 19) launch_chained(kernel, grid, block, smem, st, std::forward<Args>(args)...);
    else launch(kernel, grid, block, smem, st, std::forward<Args>(args)...);
}

constexpr int kQuads = 5;        // 16-byte quads (two pairs) per label
constexpr int kPairs = 9;        // pairs (lo[b+1], up[b])
constexpr int kOrdWarps = 4;     // warps per block of the splat and bins kernels
constexpr int kOrdThreads = 32 * kOrdWarps;
constexpr int kOrdBlockMaxL = 160;  // labels of the dense form's long lists at most (its ring's shared memory)

// Mask words per vertex; labels 32 j .. 32 j + 31 are words 5 j .. 5 j + 4.
__host__ __device__ constexpr int ord_words(int L) { return (kQuads * L + 31) / 32; }
// A pixel's bins: c_lower << 8 | c_upper per label, rows of 16-byte multiples.
__host__ __device__ constexpr int ord_bin_row(int L) { return (L + 7) & ~7; }

// Row of the up[0] plane, in floats.
__host__ __device__ constexpr int ord_plane_row(int L) { return (L + 3) & ~3; }

// ---------------------------------------------------------------- bins --
// quads_of: cmax, the largest lower bin of a (vertex, label)'s entries, decides
// which of its quads some entry reaches.
__device__ __forceinline__ int quads_of(int cmax) { return (cmax + 1) >> 1; }

// Bins of Q, or of rescale(Q) (RESCALE: (Q - min) / (max - min) with min / max
// at qmm[0..1], src/eigen_utils.cpp:120-141): a tile of pixels per warp, staged
// like the plain filter's rows.  Labels past L get bin 0.  pmask: the quads a
// pixel's bins reach, as mask words [N][NW]; a vertex's mask is the or of its
// entries'.
constexpr int kBinTile = 32;
constexpr int kBinTileMaxL = 96;  // four warps' tiles in 48 KB (97 labels, 320x240: 479 us by tiles, 484 wide)

template <bool RESCALE>
__global__ void __launch_bounds__(kOrdThreads)
    ord_bins_kernel(int N, int L, const float* __restrict__ Q, const float* __restrict__ qmm,
                    uint4* __restrict__ bins, unsigned* __restrict__ pmask, int vec) {
    extern __shared__ __align__(16) unsigned char bin_smem[];
    const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float* buf = reinterpret_cast<float*>(bin_smem) + (size_t)wib * ((kBinTile * L + 3) & ~3);
    grid_release();
    grid_wait();
    const long p0 = ((long)blockIdx.x * kOrdWarps + wib) * kBinTile;
    if (p0 >= N) return;  // warp-uniform, no barrier follows
    const int np = (int)min((long)kBinTile, N - p0);
    const long t0 = p0 * L;  // a multiple of 4
    const int ne = np * L, n4 = vec ? ne >> 2 : 0;
    for (int e = lane; e < n4; e += 32) cp_async16(buf + 4 * e, Q + t0 + 4 * e);
    for (int e = 4 * n4 + lane; e < ne; e += 32) cp_async4(buf + e, Q + t0 + e);
    cp_async_commit();
    float mn = 0.0f, range = 0.0f;
    if (RESCALE) {
        mn = qmm[0];
        range = fsub(qmm[1], qmm[0]);
    }
    cp_async_wait<0>();
    __syncwarp();
    // in place: this lane's elements become their bins ...
    for (int e = lane; e < ne; e += 32) {
        float q = buf[e];
        if (RESCALE) {
            q = fsub(q, mn);
            if (range > 0.0f) q = q / range;
        }
        buf[e] = __int_as_float(bin_lower(q) << 8 | bin_upper(q));
    }
    __syncwarp();
    if (lane < np) {
        const int* b = reinterpret_cast<const int*>(buf) + lane * L;
        unsigned* pm = pmask + (p0 + lane) * ord_words(L);
        unsigned long long acc = 0;
        int have = 0;
        for (int k = 0; k < L; k++) {
            acc |= (unsigned long long)((1u << quads_of(b[k] >> 8)) - 1u) << have;
            have += kQuads;
            if (have >= 32) {
                *pm++ = (unsigned)acc;
                acc >>= 32;
                have -= 32;
            }
        }
        if (have) *pm = (unsigned)acc;
    }
    // ... and rows of 8 labels leave 16 bytes at a time
    const int G = ord_bin_row(L) / 8;
    for (int it = lane; it < np * G; it += 32) {
        const int pl = it / G, k0 = 8 * (it - pl * G);
        const int* b = reinterpret_cast<const int*>(buf) + pl * L + k0;
        unsigned w[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const unsigned lo = k0 + 2 * i < L ? b[2 * i] : 0, hi = k0 + 2 * i + 1 < L ? b[2 * i + 1] : 0;
            w[i] = lo | hi << 16;
        }
        bins[p0 * G + it] = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// Bins of Q for any number of labels, without shared memory: a warp per pixel,
// 32 labels at a time (lane = label, their 160 mask bits five words of their
// own), the label blocks shared by gridDim.y warps where the pixels are few.
// The whole filter with the tiles above in up to 227 KB, which ended at 454
// labels, -> this: 320x240, five features, 150 labels 660 -> 651 us, 300 1218 ->
// 1147; 160x120, 454 labels 803 -> 765; 64x48, 128 labels 131 -> 123.
__global__ void __launch_bounds__(kOrdThreads)
    ord_bins_wide_kernel(int N, int L, const float* __restrict__ Q, unsigned short* __restrict__ bins,
                         unsigned* __restrict__ pmask) {
    const int lane = threadIdx.x & 31, nblk = (L + 31) / 32, Lb = ord_bin_row(L), NW = ord_words(L);
    grid_release();
    grid_wait();
    const long i = (long)blockIdx.x * kOrdWarps + (threadIdx.x >> 5);
    if (i >= N) return;  // warp-uniform
    const int at = kQuads * lane & 31, word = kQuads * lane >> 5;  // this lane's mask bits
    for (int blk = blockIdx.y; blk < nblk; blk += gridDim.y) {
        const int k = 32 * blk + lane;
        const float q = k < L ? Q[i * L + k] : 0.0f;
        const int cl = bin_lower(q);
        if (k < Lb) bins[i * Lb + k] = (unsigned short)(cl << 8 | bin_upper(q));
        const unsigned long long bits = (unsigned long long)((1u << quads_of(cl)) - 1u) << at;
        const unsigned lo = (unsigned)bits, hi = (unsigned)(bits >> 32);
        unsigned mine = 0;
#pragma unroll
        for (int r = 0; r < kQuads; r++) {
            const unsigned w = __reduce_or_sync(0xffffffffu, word == r ? lo : word + 1 == r ? hi : 0u);
            if (lane == r) mine = w;
        }
        if (lane < kQuads && kQuads * blk + lane < NW) pmask[i * NW + kQuads * blk + lane] = mine;
    }
}

// --------------------------------------------------------------- splat --
// The quad count of this lane's label from the words (lane r < 5 holds word r).
__device__ __forceinline__ int mask_quads(unsigned word, int lane) {
    const int idx = kQuads * lane, w0 = idx >> 5, sh = idx & 31;
    const unsigned lo = __shfl_sync(0xffffffffu, word, w0), hi = __shfl_sync(0xffffffffu, word, min(w0 + 1, 31));
    return __popc(__funnelshift_r(lo, hi, sh) & ((1u << kQuads) - 1u));
}

// Long lists, first pass: the masks, the or of the entries' pixel masks.  A
// block per list; the order does not matter, so its warps take entries in turn.
constexpr int kMaskWarps = 4;
template <int NWC>
__global__ void __launch_bounds__(32 * kMaskWarps)
    ord_mask_kernel(int NWr, const int* __restrict__ order, const int* __restrict__ seg_start,
                    const int2* __restrict__ seg, const unsigned* __restrict__ pmask, unsigned* __restrict__ act) {
    const int NW = NWC ? NWC : NWr, t = threadIdx.x, lane = t & 31;
    __shared__ unsigned red[kMaskWarps];
    __shared__ uint4 red4[kMaskWarps];
    grid_release();
    grid_wait();
    const int v = order[blockIdx.x];
    const int s0 = seg_start[v], s1 = seg_start[v + 1];
    if (NWC == 4) {
        uint4 m = make_uint4(0, 0, 0, 0);
#pragma unroll 4
        for (int s = s0 + t; s < s1; s += 32 * kMaskWarps) {
            const uint4 x = *reinterpret_cast<const uint4*>(pmask + 4 * (long)seg[s].x);
            m.x |= x.x;
            m.y |= x.y;
            m.z |= x.z;
            m.w |= x.w;
        }
        m.x = __reduce_or_sync(0xffffffffu, m.x);
        m.y = __reduce_or_sync(0xffffffffu, m.y);
        m.z = __reduce_or_sync(0xffffffffu, m.z);
        m.w = __reduce_or_sync(0xffffffffu, m.w);
        if (lane == 0) red4[t >> 5] = m;
        __syncthreads();
        if (t == 0) {
            for (int w = 1; w < kMaskWarps; w++) {
                m.x |= red4[w].x;
                m.y |= red4[w].y;
                m.z |= red4[w].z;
                m.w |= red4[w].w;
            }
            *reinterpret_cast<uint4*>(act + 4 * (long)(v + 1)) = m;
        }
    } else {
        for (int r = 0; r < NW; r++) {
            unsigned m = 0;
            for (int s = s0 + t; s < s1; s += 32 * kMaskWarps) m |= pmask[(long)seg[s].x * NW + r];
            m = __reduce_or_sync(0xffffffffu, m);
            if (lane == 0) red[t >> 5] = m;
            __syncthreads();
            if (t == 0) {
                for (int w = 1; w < kMaskWarps; w++) m |= red[w];
                act[(long)(v + 1) * NW + r] = m;
            }
            __syncthreads();
        }
    }
}

// The bins of one entry as floats offset by 2^23 (exact: one byte permute
// each), and P pairs b0 .. b0 + P - 1 of one entry: masks [c_lower > b] =
// sat(c_lower - b) and [c_upper <= b] = sat(b + 1 - c_upper), exactly 0 or 1
// for these small integers, then one f32x2 FMA: fma(1, w, acc) rounds acc + w
// once, fma(0, w, acc) is acc (a sum is never -0: it starts at +0).
template <int P>
struct PairSums {
    unsigned long long acc[P];
    float nlo[P], up[P];
    __device__ __forceinline__ void init(int b0) {
#pragma unroll
        for (int i = 0; i < P; i++) {
            acc[i] = 0ull;
            nlo[i] = -(8388608.0f + (float)(b0 + i));
            up[i] = 8388608.0f + (float)(b0 + i + 1);
        }
    }
    __device__ __forceinline__ void add(unsigned c, unsigned long long w2) {
        const float cl = __uint_as_float(__byte_perm(c, 0x4b000000u, 0x7541));
        const float cu = __uint_as_float(__byte_perm(c, 0x4b000000u, 0x7540));
#pragma unroll
        for (int i = 0; i < P; i++)
            asm("{\n\t.reg .f32 ml, mu;\n\t.reg .b64 m;\n\t"
                "add.rn.sat.f32 ml, %1, %3;\n\t"
                "sub.rn.sat.f32 mu, %4, %2;\n\t"
                "mov.b64 m, {ml, mu};\n\t"
                "fma.rn.f32x2 %0, m, %5, %0;\n\t}"
                : "+l"(acc[i])
                : "f"(cl), "f"(cu), "f"(nlo[i]), "f"(up[i]), "l"(w2));
    }
    __device__ __forceinline__ void store(float* label, int b0) {
#pragma unroll
        for (int i = 0; i < P; i++)
            if (b0 + i < kPairs) *reinterpret_cast<unsigned long long*>(label + 2 * (b0 + i)) = acc[i];
    }
};

// Units of P pairs that cover nq quads.
template <int P>
__device__ __forceinline__ int units_of(int nq) {
    return min((kPairs + P - 1) / P, (2 * nq + P - 1) / P);
}

// Appends this lane's n units (tag | u) to list at `at`, after those of the
// lanes before it; returns the new length (warp-uniform).
__device__ __forceinline__ int append_units(unsigned short* list, int at, int n, int tag, int lane) {
    int x = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    for (int u = 0; u < n; u++) list[at + x - n + u] = (unsigned short)(tag | u);
    return at + __shfl_sync(0xffffffffu, x, 31);
}

// Warp instructions per entry of a round of units of P pairs (see PairSums::add:
// one 2-byte and half a 16-byte shared-memory read, two byte permutes, 2 P
// saturated adds and P packed FMAs), times two.
__device__ __forceinline__ int round_cost(int P) { return 2 * (3 * P) + 7; }

// Long lists, second pass: one warp per (list, block of 32 labels, 32 units),
// a unit being P pairs of one label.  The list's bins (16 bytes per 8 labels)
// stream through a ring of kOrdStages chunks of 32 entries by cp.async; each
// lane adds its unit's pairs entry by entry.  P is 2 or 3, whichever needs
// fewer instructions for the list's mask (few bins reached: 21 units of two
// pairs fit one round; all of them: 63 units of three fit two), but 1 for the
// longest lists (over kHugeList entries): their single chain sets the launch's
// length, and it is half as long.
constexpr int kOrdStages = 4;
// bytes of one ring per warp: bins of at most 32 labels, (w, w) pairs; + the unit list
__host__ __device__ constexpr int ord_ring_bytes(int nc) { return kOrdStages * 32 * (nc * 16 + 8); }
constexpr int kUnitList = 32 * kPairs;  // units of 32 labels at most

// NC: 16-byte groups per entry as a compile-time constant (L <= 32), or 0.
constexpr int kLongRounds = 5;  // rounds of 32 units that 32 labels can need: 160 of P = 2
template <int P, int NC>
__device__ __forceinline__ void ord_long_round(int round, int blk, int v, int nq, int L,
                                               const int* __restrict__ seg_start, const int2* __restrict__ seg,
                                               const uint4* __restrict__ bins, float* __restrict__ vals,
                                               unsigned char* smem, int lane) {
    const int G = ord_bin_row(L) / 8;
    unsigned short* list = reinterpret_cast<unsigned short*>(smem);
    const int A = append_units(list, 0, units_of<P>(nq), lane << 4, lane);
    if (32 * round >= A) return;  // warp-uniform
    __syncwarp();
    const int i = 32 * round + lane;
    const bool on = i < A;
    const int k = on ? list[i] >> 4 : 0, b0 = on ? P * (list[i] & 15) : 0;
    const int s0 = seg_start[v], s1 = seg_start[v + 1], nch = (s1 - s0 + 31) >> 5;
    const int g0 = 4 * blk, nc = NC ? NC : min(4, G - g0);
    uint4* X = reinterpret_cast<uint4*>(smem + 2 * kUnitList);                      // [stage][entry][nc]
    float2* Wt = reinterpret_cast<float2*>(X + kOrdStages * 32 * nc);               // [stage][entry]
    auto entry = [&](int c) {  // this lane's entry of chunk c; weight 0 past the end
        const int s = s0 + c * 32 + lane;
        return (c < nch && s < s1) ? seg[s] : make_int2(0, 0);
    };
    auto issue = [&](int c, int2 e) {
        if (c < nch) {
            const int slot = c % kOrdStages, n = min(32, s1 - (s0 + c * 32));
#pragma unroll
            for (int j = 0; j < (NC ? NC : 4); j++) {
                if (!NC && j >= nc) break;
                const int idx = lane + 32 * j, en = idx / nc;
                const int p = __shfl_sync(0xffffffffu, e.x, en);
                if (en < n) cp_async16(X + slot * 32 * nc + idx, bins + (long)p * G + g0 + (idx - en * nc));
            }
            const float w = entry_w(e);
            Wt[slot * 32 + lane] = make_float2(w, w);
        }
        cp_async_commit();
    };
    PairSums<P> ps;
    ps.init(b0);
    int2 e0 = entry(0), e1 = entry(1);
#pragma unroll
    for (int c = 0; c < kOrdStages - 1; c++) {
        issue(c, e0);
        e0 = e1;
        e1 = entry(c + 2);
    }
    for (int c = 0; c < nch; c++) {
        cp_async_wait<kOrdStages - 2>();
        __syncwarp();
        const int slot = c % kOrdStages;
        const unsigned short* xs = reinterpret_cast<const unsigned short*>(X + slot * 32 * nc) + k;
        const ulonglong2* ws = reinterpret_cast<const ulonglong2*>(Wt + slot * 32);
#pragma unroll 8
        for (int e = 0; e < 32; e += 2) {
            const ulonglong2 w = ws[e >> 1];
            ps.add(xs[e * 8 * nc], w.x);
            ps.add(xs[(e + 1) * 8 * nc], w.y);
        }
        __syncwarp();  // the next issue refills the slot of chunk c - 1 .. c
        issue(c + kOrdStages - 1, e0);
        e0 = e1;
        e1 = entry(c + kOrdStages + 1);
    }
    cp_async_wait<0>();
    if (on) ps.store(vals + (long)(v + 1) * kOrdW * L + (long)(32 * blk + k) * kOrdW, b0);
}

// Tasks run over the lists first, then over their rounds: the first rounds,
// which every list has, fill whole blocks, and most later ones exit at once (a
// list's rounds side by side in a block left three of its four warps idle).
template <bool HUGE, int NC>
__device__ __forceinline__ void ord_splat_long(int task, int lists, int nblk, int L, int NW, const int* __restrict__ order,
                                               const int* __restrict__ seg_start, const int2* __restrict__ seg,
                                               const uint4* __restrict__ bins, const unsigned* __restrict__ act,
                                               float* __restrict__ vals, unsigned char* smem, int lane) {
    const int round = task / (lists * nblk), rest = task - round * (lists * nblk);
    const int li = rest / nblk, blk = rest - li * nblk;
    const int v = order[li];
    const int cnt = min(kQuads, NW - kQuads * blk);
    const unsigned word = lane < cnt ? act[(long)(v + 1) * NW + kQuads * blk + lane] : 0u;
    const int nq = mask_quads(word, lane);
    if (HUGE) {
        ord_long_round<1, NC>(round, blk, v, nq, L, seg_start, seg, bins, vals, smem, lane);
        return;
    }
    const int r2 = (__reduce_add_sync(0xffffffffu, units_of<2>(nq)) + 31) >> 5,
              r3 = (__reduce_add_sync(0xffffffffu, units_of<3>(nq)) + 31) >> 5;
    if (round >= max(r2, r3)) return;  // warp-uniform
    if (r2 * round_cost(2) <= r3 * round_cost(3))
        ord_long_round<2, NC>(round, blk, v, nq, L, seg_start, seg, bins, vals, smem, lane);
    else
        ord_long_round<3, NC>(round, blk, v, nq, L, seg_start, seg, bins, vals, smem, lane);
}

// Short lists: a warp takes four consecutive ones (as many as fit in
// kGroupEntries entries at a time), finds their masks and adds their units of P
// pairs (2 or 3, as for the long lists), packed into lanes across the four:
// with few labels active a vertex has a handful of units, and one warp would
// idle on it.  All entries' (pixel, weight), then all their masks and bins, are
// in flight together: the warp waits for memory five times, not once per list
// and per eight entries.
constexpr int kGroup = 4;
constexpr int kGroupEntries = 128;  // at least two lists of kLongList
constexpr int kGroupList = kGroup * 32 * kQuads;
__host__ __device__ constexpr int ord_group_bytes(int nc) { return kGroupEntries * (nc * 16 + 8) + 2 * kGroupList; }
struct GroupLists {
    int at[kGroup + 1], v[kGroup], nq[kGroup], m;
};
template <int P>
__device__ __forceinline__ void ord_group_rounds(const GroupLists& g, int blk, int L, int stride,
                                                 const unsigned short* xs, const int2* E, unsigned short* list,
                                                 float* __restrict__ vals, int lane) {
    int A = 0;
#pragma unroll
    for (int j = 0; j < kGroup; j++)
        if (j < g.m) A = append_units(list, A, units_of<P>(g.nq[j]), j << 9 | lane << 4, lane);
    __syncwarp();
    for (int i0 = 0; i0 < A; i0 += 32) {
        const int i = i0 + lane;
        const bool on = i < A;
        const int t = on ? list[i] : 0;
        const int j = t >> 9, k = t >> 4 & 31, b0 = P * (t & 15);
        int a0 = g.at[0], n = g.at[1] - g.at[0], vv = g.v[0];
#pragma unroll
        for (int q = 1; q < kGroup; q++)
            if (j == q) {
                a0 = g.at[q];
                n = g.at[q + 1] - g.at[q];
                vv = g.v[q];
            }
        if (!on) n = 0;
        const int nmax = __reduce_max_sync(0xffffffffu, n), last = max(n - 1, 0);
        PairSums<P> ps;
        ps.init(b0);
        const unsigned short* x = xs + a0 * stride + k;
        const int2* en = E + a0;
#pragma unroll 4
        for (int e = 0; e < nmax; e++) {  // past a lane's list: its last entry with weight 0, which adds nothing
            const int ee = min(e, last);
            const float w = e < n ? entry_w(en[ee]) : 0.0f;
            ps.add(x[ee * stride], pack2(w, w));
        }
        if (on) ps.store(vals + (long)(vv + 1) * kOrdW * L + (long)(32 * blk + k) * kOrdW, b0);
    }
    __syncwarp();  // list is refilled
}

template <int NC, int NWC>
__device__ __forceinline__ void ord_splat_group(int first, int count, int L, int NWr, const int* __restrict__ order,
                                                const int* __restrict__ seg_start, const int2* __restrict__ seg,
                                                const uint4* __restrict__ bins, const unsigned* __restrict__ pmask,
                                                unsigned* __restrict__ act, float* __restrict__ vals,
                                                unsigned char* smem, int lane) {
    const int G = ord_bin_row(L) / 8, NW = NWC ? NWC : NWr;
    constexpr int kI = kGroupEntries / 32;
    unsigned short* list = reinterpret_cast<unsigned short*>(smem);
    int2* E = reinterpret_cast<int2*>(smem + 2 * kGroupList);  // [entry] (pixel, weight)
    uint4* X = reinterpret_cast<uint4*>(E + kGroupEntries);    // [entry][nc] bins
    // lane j < count: list j's vertex, start and length
    const int vj = lane < count ? order[first + lane] : 0;
    const int sj = lane < count ? seg_start[vj] : 0, nj = lane < count ? seg_start[vj + 1] - sj : 0;
    for (int j0 = 0; j0 < count;) {
        GroupLists g;
        int start[kGroup];  // the lists j0 .. j0 + m - 1 of this round
        g.m = 0;
        g.at[0] = 0;
#pragma unroll
        for (int j = 0; j < kGroup; j++) {
            const int src = min(j0 + j, 31);
            const int n = __shfl_sync(0xffffffffu, nj, src);
            g.v[j] = __shfl_sync(0xffffffffu, vj, src);
            start[j] = __shfl_sync(0xffffffffu, sj, src);
            const bool take = g.m == j && j0 + j < count && g.at[j] + n <= kGroupEntries;
            g.at[j + 1] = g.at[j] + (take ? n : 0);
            g.m += take;
        }
        const int tot = g.at[kGroup];
        int jl[kI];  // this lane's entries lane + 32 i: their list, or kGroup
        int2 ent[kI];
#pragma unroll
        for (int i = 0; i < kI; i++) {
            const int t = lane + 32 * i;
            jl[i] = kGroup;
            ent[i] = make_int2(0, 0);
            if (t < tot) {
                int j = 0, s = start[0];
#pragma unroll
                for (int q = 1; q < kGroup; q++)
                    if (t >= g.at[q]) {
                        j = q;
                        s = start[q] - g.at[q];
                    }
                jl[i] = j;
                ent[i] = seg[s + t];
            }
        }
        __syncwarp();  // E and X are free
#pragma unroll
        for (int i = 0; i < kI; i++) E[lane + 32 * i] = ent[i];
        __syncwarp();
        for (int blk = 0; 32 * blk < L; blk++) {
            const int g0 = 4 * blk, nc = NC ? NC : min(4, G - g0);
            for (int idx = lane; idx < tot * nc; idx += 32) {
                const int en = idx / nc;
                cp_async16(X + idx, bins + (long)E[en].x * G + g0 + (idx - en * nc));
            }
            cp_async_commit();
            // the masks meanwhile: lane r < 5 ends with word r of list j, then its label's quads
            unsigned word[kGroup] = {0, 0, 0, 0};
            auto reduce = [&](int r, const unsigned (&x)[kI]) {
#pragma unroll
                for (int j = 0; j < kGroup; j++) {
                    unsigned y = 0;
#pragma unroll
                    for (int i = 0; i < kI; i++) y |= jl[i] == j ? x[i] : 0u;
                    y = __reduce_or_sync(0xffffffffu, y);
                    if (lane == r) word[j] = y;
                }
            };
            if (NWC == 4) {
                uint4 x[kI];
#pragma unroll
                for (int i = 0; i < kI; i++)
                    x[i] = *reinterpret_cast<const uint4*>(pmask + 4 * (long)ent[i].x);  // an idle slot: pixel 0, unused
                const unsigned xa[kI] = {x[0].x, x[1].x, x[2].x, x[3].x}, xb[kI] = {x[0].y, x[1].y, x[2].y, x[3].y},
                               xc[kI] = {x[0].z, x[1].z, x[2].z, x[3].z}, xd[kI] = {x[0].w, x[1].w, x[2].w, x[3].w};
                reduce(0, xa);
                reduce(1, xb);
                reduce(2, xc);
                reduce(3, xd);
            } else {
                for (int r = 0; r < kQuads && kQuads * blk + r < NW; r++) {
                    unsigned x[kI];
#pragma unroll
                    for (int i = 0; i < kI; i++) x[i] = pmask[(long)ent[i].x * NW + kQuads * blk + r];
                    reduce(r, x);
                }
            }
            int u2 = 0, u3 = 0;
#pragma unroll
            for (int j = 0; j < kGroup; j++) {
                g.nq[j] = 0;
                if (j < g.m) {  // warp-uniform
                    if (lane < kQuads && kQuads * blk + lane < NW)
                        act[(long)(g.v[j] + 1) * NW + kQuads * blk + lane] = word[j];
                    g.nq[j] = mask_quads(word[j], lane);
                }
                u2 += units_of<2>(g.nq[j]);
                u3 += units_of<3>(g.nq[j]);
            }
            const int r2 = (__reduce_add_sync(0xffffffffu, u2) + 31) >> 5,
                      r3 = (__reduce_add_sync(0xffffffffu, u3) + 31) >> 5;
            cp_async_wait<0>();
            __syncwarp();
            const unsigned short* xs = reinterpret_cast<const unsigned short*>(X);
            if (r2 * round_cost(2) <= r3 * round_cost(3))
                ord_group_rounds<2>(g, blk, L, 8 * nc, xs, E, list, vals, lane);
            else
                ord_group_rounds<3>(g, blk, L, 8 * nc, xs, E, list, vals, lane);
        }
        j0 += g.m;
    }
}

// Very short lists: a thread per (list, label), all nine pairs in registers, the
// next entry's loads in flight; thread k < NW of a list also finds mask word k.  A
// group of four lists of three entries each leaves its warp mostly idle (a noisy
// 640x480 image: one label 447 -> 263 us the filter, 4 1069 -> 929; 320x240, 12
// labels 589 -> 571).
__device__ __forceinline__ void ord_splat_few(long t, int n_short, int L, int NW, const int* __restrict__ order,
                                              const int* __restrict__ seg_start, const int2* __restrict__ seg,
                                              const unsigned short* __restrict__ bins,
                                              const unsigned* __restrict__ pmask, unsigned* __restrict__ act,
                                              float* __restrict__ vals) {
    if (t >= (long)n_short * L) return;
    const int u = (int)(t / L), k = (int)(t - (long)u * L), Lb = ord_bin_row(L);
    const int v = order[u], s0 = seg_start[v], s1 = seg_start[v + 1];
    PairSums<kPairs> ps;
    ps.init(0);
    unsigned m = 0;
    int cmax = 0;
#pragma unroll 2
    for (int s = s0; s < s1; s++) {
        const int2 e = seg[s];
        const unsigned c = bins[(long)e.x * Lb + k];
        if (k < NW) m |= pmask[(long)e.x * NW + k];
        cmax = max(cmax, (int)(c >> 8));
        ps.add(c, pack2(entry_w(e), entry_w(e)));
    }
    if (k < NW) act[(long)(v + 1) * NW + k] = m;
    unsigned long long* label = reinterpret_cast<unsigned long long*>(vals + (long)(v + 1) * kOrdW * L + (long)k * kOrdW);
    const int n = 2 * quads_of(cmax);
#pragma unroll
    for (int i = 0; i < kPairs; i++)
        if (i < n) label[i] = ps.acc[i];
}

// One launch: warps [0, huge_tasks) the lists over kHugeList entries, the next
// long_tasks the other long ones (longest first), the rest groups of short
// lists, or (FEW) 32 (list, label) of them each.  Row 0 of both masks (the absent neighbour) is cleared here: none of
// its quads exists, and its T is 0.
template <int NC, int NWC, bool FEW>
__global__ void __launch_bounds__(kOrdThreads, 6)
    ord_splat_kernel(int M, int n_long, int n_huge, int huge_tasks, int long_tasks, int L, int NW,
                     const int* __restrict__ order, const int* __restrict__ seg_start, const int2* __restrict__ seg,
                     const uint4* __restrict__ bins, const unsigned* __restrict__ pmask, unsigned* __restrict__ act,
                     unsigned* __restrict__ act2, float* __restrict__ vals, int warp_bytes) {
    extern __shared__ __align__(16) unsigned char ord_smem[];
    const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned char* smem = ord_smem + (size_t)wib * warp_bytes;
    grid_release();
    grid_wait();
    if (blockIdx.x == 0)
        for (int r = threadIdx.x; r < NW; r += blockDim.x) act[r] = act2[r] = 0u;
    const int nblk = (L + 31) / 32;
    long t = (long)blockIdx.x * kOrdWarps + wib;
    if (t < huge_tasks) {
        ord_splat_long<true, NC>((int)t, n_huge, nblk, L, NW, order, seg_start, seg, bins, act, vals, smem, lane);
        return;
    }
    t -= huge_tasks;
    if (t < long_tasks) {
        ord_splat_long<false, NC>((int)t, n_long - n_huge, nblk, L, NW, order + n_huge, seg_start, seg, bins, act, vals, smem, lane);
        return;
    }
    t -= long_tasks;
    if (FEW) {
        ord_splat_few(32 * t + lane, M - n_long, L, NW, order + n_long, seg_start, seg,
                      reinterpret_cast<const unsigned short*>(bins), pmask, act, vals);
        return;
    }
    const long first = n_long + t * kGroup;
    if (first < M)
        ord_splat_group<NC, NWC>((int)first, (int)min((long)kGroup, M - first), L, NW, order, seg_start, seg, bins,
                                 pmask, act, vals, smem, lane);
}

// ---------------------------------------------------------------- blur --
// A quad of a source row where it is stored; r keeps (0, T, 0, T) where no entry
// reached it.
__device__ __forceinline__ void quad_if(float4& r, const float4* p, bool stored) {
    asm("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %5, 0;\n\t"
        "@p ld.global.v4.f32 {%0, %1, %2, %3}, [%4];\n\t}"
        : "+f"(r.x), "+f"(r.y), "+f"(r.z), "+f"(r.w)
        : "l"(p), "r"((unsigned)stored));
}

// One axis, weightedAddSplitArray (:570-578): a warp per vertex, lane = quad, 32
// quads (a mask word) at a time.  The result has the quads of the vertex or of
// either neighbour; only stored quads are read.  The chain neighbours -> masks
// -> quads is three loads long, so a grid that fills the SMs walks the vertices
// and loads each step's neighbours two steps, its masks and T one step ahead.
// LAST: what the slice reads is completed: the plane up[0] of every label (T
// where the quad does not exist), contiguous over labels; up[9] = T beside
// pair 8; and behind a label's last stored quad one more of (0, T, 0, T), so
// that up[c] of an entry in bin c is there whichever quad it falls in.
// NWC: mask words as a compile-time constant (1 .. 4: up to 6, 12, 19, 25 labels),
// or 0 (two at a time).  152x71, 18 labels: 5.6 us as a loop over single words.
constexpr int kOrdBlurThreads = 256;
constexpr int kOrdBlurBlocks = 3;  // per SM
template <int NWC, bool LAST>
__global__ void __launch_bounds__(kOrdBlurThreads, kOrdBlurBlocks)
    ord_blur_kernel(int M, int L, int NWr, const int2* __restrict__ nbr, const float* __restrict__ T,
                    const float* __restrict__ Tn, const float4* __restrict__ src, float4* __restrict__ dst,
                    const unsigned* __restrict__ act, unsigned* __restrict__ act2, float* __restrict__ plane) {
    const int NW = NWC ? NWC : NWr, row4 = kQuads * L;
    const int lane = threadIdx.x & 31;
    const int nw = gridDim.x * (kOrdBlurThreads / 32);
    int v = blockIdx.x * (kOrdBlurThreads / 32) + (threadIdx.x >> 5);
    grid_release();
    grid_wait();
    struct Quads {
        float4 x, y, z;
    };
    struct Sources {  // the rows of a vertex and its neighbours, and their T
        const float4 *p0, *p1, *p2;
        float T0, T1, T2;
    };
    auto load = [&](const Sources& s, int r, unsigned a, unsigned b, unsigned c, Quads& q) {
        q.x = make_float4(0.0f, s.T0, 0.0f, s.T0);
        q.y = make_float4(0.0f, s.T1, 0.0f, s.T1);
        q.z = make_float4(0.0f, s.T2, 0.0f, s.T2);
        quad_if(q.x, s.p0 + 32 * r, a >> lane & 1u);
        quad_if(q.y, s.p1 + 32 * r, b >> lane & 1u);
        quad_if(q.z, s.p2 + 32 * r, c >> lane & 1u);
    };
    // m: this word's result mask, before: the previous word's (LAST)
    auto store = [&](const Quads& s, int vv, int r, unsigned m, unsigned before, float Tl) {
        bool on = m >> lane & 1u;
        float4 q;
        q.x = fadd(s.x.x, fmul(0.5f, fadd(s.y.x, s.z.x)));
        q.y = fadd(s.x.y, fmul(0.5f, fadd(s.y.y, s.z.y)));
        q.z = fadd(s.x.z, fmul(0.5f, fadd(s.y.z, s.z.z)));
        q.w = fadd(s.x.w, fmul(0.5f, fadd(s.y.w, s.z.w)));
        const int idx = 32 * r + lane;
        if (LAST) {
            const int k = idx / kQuads, j = idx - k * kQuads;
            const unsigned bm = m << 1 | before >> 31;  // the quad before this one
            if (j == kQuads - 1) q.w = Tl;
            if (k < L && j == 0) plane[(long)(vv + 1) * ord_plane_row(L) + k] = q.y;
            on = on || (k < L && j > 0 && (bm >> lane & 1u));
        }
        if (on) dst[(long)(vv + 1) * row4 + idx] = q;
    };
    if (NWC == 4) {
        const uint4* act4 = reinterpret_cast<const uint4*>(act);
        uint4 a, b, c;
        Sources s;
        float Tl = 0.0f;
        auto fetch = [&](int vv, int2 nb) {  // masks, T and row pointers of vertex vv
            a = act4[vv + 1];
            b = act4[nb.x];
            c = act4[nb.y];
            s.T0 = T[vv + 1];
            s.T1 = T[nb.x];
            s.T2 = T[nb.y];
            if (LAST) Tl = Tn[vv + 1];
            s.p0 = src + (long)(vv + 1) * row4 + lane;
            s.p1 = src + (long)nb.x * row4 + lane;
            s.p2 = src + (long)nb.y * row4 + lane;
        };
        if (v >= M) return;
        fetch(v, nbr[v]);
        int2 nb = nbr[min(v + nw, M - 1)];
        for (; v < M; v += nw) {
            const uint4 m = make_uint4(a.x | b.x | c.x, a.y | b.y | c.y, a.z | b.z | c.z, a.w | b.w | c.w);
            Quads q0, q1;
            load(s, 0, a.x, b.x, c.x, q0);
            load(s, 1, a.y, b.y, c.y, q1);
            const Sources cur = s;
            const uint4 ca = a, cb = b, cc = c;
            const float cT = Tl;
            fetch(min(v + nw, M - 1), nb);
            nb = nbr[min(v + 2 * nw, M - 1)];
            store(q0, v, 0, m.x, 0u, cT);
            load(cur, 2, ca.z, cb.z, cc.z, q0);
            store(q1, v, 1, m.y, m.x, cT);
            load(cur, 3, ca.w, cb.w, cc.w, q1);
            if (!LAST && lane == 0) reinterpret_cast<uint4*>(act2)[v + 1] = m;
            store(q0, v, 2, m.z, m.y, cT);
            store(q1, v, 3, m.w, m.z, cT);
        }
    } else {
        constexpr int C = NWC ? NWC : 2;  // words at a time: all of them, or two
        unsigned a[C], b[C], c[C];
        Sources s;
        float Tl = 0.0f;
        auto masks = [&](int vv, int2 nb, int r0) {
#pragma unroll
            for (int i = 0; i < C; i++) {
                const bool in = NWC || r0 + i < NW;
                a[i] = in ? act[(long)(vv + 1) * NW + r0 + i] : 0u;
                b[i] = in ? act[(long)nb.x * NW + r0 + i] : 0u;
                c[i] = in ? act[(long)nb.y * NW + r0 + i] : 0u;
            }
        };
        auto fetch = [&](int vv, int2 nb) {  // the first masks, T and row pointers of vertex vv
            masks(vv, nb, 0);
            s.T0 = T[vv + 1];
            s.T1 = T[nb.x];
            s.T2 = T[nb.y];
            if (LAST) Tl = Tn[vv + 1];
            s.p0 = src + (long)(vv + 1) * row4 + lane;
            s.p1 = src + (long)nb.x * row4 + lane;
            s.p2 = src + (long)nb.y * row4 + lane;
        };
        if (v >= M) return;
        int2 nb = nbr[v];
        fetch(v, nb);
        int2 nn = nbr[min(v + nw, M - 1)];
        for (; v < M; v += nw) {
            const Sources cur = s;
            const float cT = Tl;
            unsigned before = 0u;
            for (int r0 = 0; r0 < NW; r0 += C) {
                unsigned m[C];
                Quads q[C];
#pragma unroll
                for (int i = 0; i < C; i++) {
                    m[i] = a[i] | b[i] | c[i];
                    load(cur, r0 + i, a[i], b[i], c[i], q[i]);
                }
                if (r0 + C < NW) {  // the next masks: this vertex's or the next one's
                    masks(v, nb, r0 + C);
                } else {
                    nb = nn;
                    fetch(min(v + nw, M - 1), nb);
                    nn = nbr[min(v + 2 * nw, M - 1)];
                }
#pragma unroll
                for (int i = 0; i < C; i++) {
                    if (!NWC && r0 + i >= NW) break;
                    if (!LAST && lane == 0) act2[(long)(v + 1) * NW + r0 + i] = m[i];
                    store(q[i], v, r0 + i, m[i], before, cT);
                    before = m[i];
                }
            }
        }
    }
}

// The same with a thread per (vertex, quad), where the quads of one mask word (up to
// 6 labels) leave a warp's lanes idle and the vertices fill the chip (from 4096 on;
// 97x83, 1100 vertices, 3 labels 16.5 us by warps, 18.8 so).  The whole filter in the quad form, a warp a
// vertex -> this, us: 640x480, five features, 2 labels 143 -> 131, a noisy image
// (650 thousand vertices) with one label 1185 -> 447, with 4 1191 -> 1069; with 8
// labels this loses, 6 to 12 %.
template <bool LAST>
__global__ void __launch_bounds__(kOrdBlurThreads)
    ord_blur_few_kernel(int M, int L, int NW, const int2* __restrict__ nbr, const float* __restrict__ T,
                        const float* __restrict__ Tn, const float4* __restrict__ src, float4* __restrict__ dst,
                        const unsigned* __restrict__ act, unsigned* __restrict__ act2, float* __restrict__ plane) {
    const int row4 = kQuads * L;
    const long t = (long)blockIdx.x * kOrdBlurThreads + threadIdx.x;
    grid_release();
    grid_wait();
    if (t >= (long)M * row4) return;
    const int v = (int)(t / row4), idx = (int)(t - (long)v * row4), r = idx >> 5, bit = idx & 31;
    const int k = idx / kQuads, j = idx - k * kQuads;
    const int2 nb = nbr[v];
    const unsigned *pa = act + (long)(v + 1) * NW + r, *pb = act + (long)nb.x * NW + r, *pc = act + (long)nb.y * NW + r;
    const unsigned a = *pa, b = *pb, c = *pc, m = a | b | c;
    if (!LAST && bit == 0) act2[(long)(v + 1) * NW + r] = m;
    bool on = m >> bit & 1u;
    if (LAST && j > 0)  // behind a stored quad
        on = on || (bit ? m >> (bit - 1) & 1u : (pa[-1] | pb[-1] | pc[-1]) >> 31);
    if (!on && !(LAST && j == 0)) return;
    const float T0 = T[v + 1], T1 = T[nb.x], T2 = T[nb.y];
    float4 x = make_float4(0.0f, T0, 0.0f, T0), y = make_float4(0.0f, T1, 0.0f, T1), z = make_float4(0.0f, T2, 0.0f, T2);
    quad_if(x, src + (long)(v + 1) * row4 + idx, a >> bit & 1u);
    quad_if(y, src + (long)nb.x * row4 + idx, b >> bit & 1u);
    quad_if(z, src + (long)nb.y * row4 + idx, c >> bit & 1u);
    float4 q;
    q.x = fadd(x.x, fmul(0.5f, fadd(y.x, z.x)));
    q.y = fadd(x.y, fmul(0.5f, fadd(y.y, z.y)));
    q.z = fadd(x.z, fmul(0.5f, fadd(y.z, z.z)));
    q.w = fadd(x.w, fmul(0.5f, fadd(y.w, z.w)));
    if (LAST) {
        if (j == kQuads - 1) q.w = Tn[v + 1];
        if (j == 0) plane[(long)(v + 1) * ord_plane_row(L) + k] = q.y;
    }
    if (on) dst[(long)(v + 1) * row4 + idx] = q;
}

// --------------------------------------------------------------- slice --
// One term of an ordered slice.
struct OrdSliceTerm {
    const int* offset;
    const float* bary;
    const float* vals;       // [(M + 1)][L][20]
    const float* T;          // blurred weight sums [M + 1]
    const float* plane;      // up[0] [(M + 1)][L]
    int d;
    float alpha;
    SliceEpilogue ep;
};

// One term's value of element (pixel, k) in any bin: the lower pass with weight
// -w alpha, then the upper with w alpha (:639-650, :687-696), one float per
// vertex and pass from the row its bin selects: T (lower bin 0), the plane up[0]
// (upper bin 0) or its pair -- the pixel's own vertices hold it.  WIDE: a row's
// bytes may not fit an int.
template <int DC, bool WIDE = false>
__device__ __forceinline__ float ord_slice_sum(const OrdSliceTerm& s, const int2* ow, int k, int cl, int cu, int L) {
    using S = std::conditional_t<WIDE, long, int>;
    const int d1 = (DC ? DC : s.d) + 1;
    const S one = sizeof(float), row = one * kOrdW * L;
    const char* lo = reinterpret_cast<const char*>(cl ? s.vals + S(k) * kOrdW + 2 * (cl - 1) : s.T);
    const char* up = reinterpret_cast<const char*>(cu ? s.vals + S(k) * kOrdW + 2 * cu + 1 : s.plane + k);
    const S ls = cl ? row : one, us = cu ? row : one * ord_plane_row(L);  // bytes
    auto at = [](const char* b, int r, S stride) {
        return *reinterpret_cast<const float*>(b + (long)r * (long)stride);
    };
    float a = 0.0f;
    if (DC) {
        float x[DC + 1], y[DC + 1];
#pragma unroll
        for (int j = 0; j <= DC; j++) {
            x[j] = at(lo, ow[j].x, ls);
            y[j] = at(up, ow[j].x, us);
        }
#pragma unroll
        for (int j = 0; j <= DC; j++) a = fadd(a, fmul(x[j], -__int_as_float(ow[j].y)));
#pragma unroll
        for (int j = 0; j <= DC; j++) a = fadd(a, fmul(y[j], __int_as_float(ow[j].y)));
    } else {
        for (int j = 0; j < d1; j++) a = fadd(a, fmul(at(lo, ow[j].x, ls), -__int_as_float(ow[j].y)));
        for (int j = 0; j < d1; j++) a = fadd(a, fmul(at(up, ow[j].x, us), __int_as_float(ow[j].y)));
    }
    return a;
}

// The slice; with two terms the second on top of the first (sa = 0 + t_0, then
// sa += t_1).  With GAP the LP's dual gap terms are folded in: tmp = (alpha +
// u) - (v + su) for the final value v, the clique term su (0 without cliques),
// and per-block sums of tmp.Q and tmp.tmp (src/densecrf.cpp:725-729).
//
// A block covers kSliceElems consecutive elements.  It stages its pixels' rows
// and weights with the bin-0 lower chain -- d+1 terms in T, the same for every
// label -- summed once per pixel; then a thread per (pixel, four labels) adds
// the plane up[0] to it with 16-byte loads, as if all were in bin 0; then the
// elements that are not (6 % in a solve) are gathered from their pairs, a
// thread each, packed.  One thread per element throughout took 122 us a solve's
// step at 640x480 (some 370 instructions and 70 L1 wavefronts per warp).
constexpr int kOsThreads = 128;
constexpr int kOsPer = 4;  // elements per thread; 1 where L < 8: the pixels' data would not fit
constexpr int kSliceElems = kOsPer * kOsThreads;
__host__ __device__ constexpr int slice_elems(int L) { return L < 8 ? kOsThreads : kSliceElems; }
// A block's dual-gap sums.
__device__ __forceinline__ void gap_store(double g0, double g1, const GapFusion& gf) {
    __shared__ double p0[kOsThreads / 32], p1[kOsThreads / 32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        g0 += __shfl_down_sync(0xffffffffu, g0, o);
        g1 += __shfl_down_sync(0xffffffffu, g1, o);
    }
    if ((threadIdx.x & 31) == 0) {
        p0[threadIdx.x >> 5] = g0;
        p1[threadIdx.x >> 5] = g1;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = 0.0, c = 0.0;
        for (int w = 0; w < kOsThreads / 32; w++) {
            a += p0[w];
            c += p1[w];
        }
        gf.partials[blockIdx.x] = a;
        gf.partials[gridDim.x + blockIdx.x] = c;
    }
}

template <bool GAP, int NT, int LC, int D0, int D1>
__global__ void __launch_bounds__(kOsThreads)
    ord_slice_kernel(int N, int Lrt, int P, OrdSliceTerm t0, OrdSliceTerm t1, const unsigned short* __restrict__ bins,
                     float* out, GapFusion gf) {
    extern __shared__ __align__(16) unsigned char os_smem[];
    __shared__ int n_hot, s_dense;
    __shared__ float s_val[kSliceElems];
    __shared__ unsigned s_hot[kSliceElems];  // element | bins << 16
    constexpr bool kWide = LC < 0;  // more labels than a block has elements, at run time as with 0
    constexpr bool kSkip = LC > 0 || (LC == 0 && D0 == 0);
    const int L = LC > 0 ? LC : Lrt, elems = slice_elems(L), Lb = ord_bin_row(L), Q = ord_plane_row(L) / 4;
    const long NL = (long)N * L, tb = (long)blockIdx.x * elems;
    const int pf = (int)(tb / L), first = (int)(tb - (long)pf * L), np = min(P, N - pf);
    const int ne = (int)min((long)elems, NL - tb);
    const int da = (D0 ? D0 : t0.d) + 1, db = (D1 ? D1 : t1.d) + 1;
    int2* s_ow[2];  // [pixel][d + 1] (row, w alpha)
    float *s_tw[2], *s_low[2], *s_nrm[2];
    s_ow[0] = reinterpret_cast<int2*>(os_smem);
    s_ow[1] = s_ow[0] + P * da;
    s_tw[0] = reinterpret_cast<float*>(s_ow[1] + (NT == 2 ? P * db : 0));
    s_tw[1] = s_tw[0] + P * da;
    s_low[0] = s_tw[1] + (NT == 2 ? P * db : 0);
    s_low[1] = s_low[0] + P;
    s_nrm[0] = s_low[1] + P;
    s_nrm[1] = s_nrm[0] + P;
    if (threadIdx.x == 0) n_hot = 0;
    grid_release();
    grid_wait();
    auto bin_of = [&](int e) {
        const int f = e + first, li = f / L;
        return (unsigned)bins[(long)(pf + li) * Lb + f - li * L];
    };
    if (threadIdx.x < 32) {  // most of a sample outside bin 0 (spread-out Q): every element on its own
        const unsigned hot = __ballot_sync(0xffffffffu, bin_of(threadIdx.x * ne / 32) != 0);
        if (threadIdx.x == 0) s_dense = __popc(hot) > 16;
    }
    float ga[kOsPer], gq[kOsPer];  // alpha + u and Q of this thread's elements, in flight meanwhile
    if (GAP) {
#pragma unroll
        for (int r = 0; r < kOsPer; r++) {
            const int e = r * kOsThreads + threadIdx.x;
            if (e < ne) {
                ga[r] = fadd(gf.alpha[tb + e], gf.u ? gf.u[tb + e] : 0.0f);
                gq[r] = gf.Q[tb + e];
            }
        }
    }
#pragma unroll
    for (int h = 0; h < NT; h++) {
        const OrdSliceTerm& s = h ? t1 : t0;
        const int d1 = h ? db : da;
        for (int e = threadIdx.x; e < np * d1; e += blockDim.x) {
            const int o = s.offset[(long)pf * d1 + e] + 1;
            const float w = fmul(s.bary[(long)pf * d1 + e], s.alpha);
            s_ow[h][e] = make_int2(o, __float_as_int(w));
            s_tw[h][e] = fmul(s.T[o], -w);
        }
        if (s.ep.norm)
            for (int e = threadIdx.x; e < np; e += blockDim.x) s_nrm[h][e] = s.ep.norm[pf + e];
    }
    __syncthreads();
    for (int e = threadIdx.x; e < NT * np; e += blockDim.x) {
        const int h = e >= np, li = e - h * np, d1 = h ? db : da;
        const float* tw = (h ? s_tw[1] : s_tw[0]) + li * d1;
        float a = 0.0f;
        for (int j = 0; j < d1; j++) a = fadd(a, tw[j]);
        (h ? s_low[1] : s_low[0])[li] = a;
    }
    __syncthreads();
    // the terms' sums a0, a1 of element (li, k) -> its value
    auto finish = [&](float a0, float a1, int li, int k) {
        const long t = (long)(pf + li) * L + k;
        float v = a0;
        if (t0.ep.potts) {
            if (t0.ep.norm) v = fmul(v, s_nrm[0][li]);
            v = t0.ep.scale_vec ? fmul(t0.ep.scale_vec[k], v) : fmul(t0.ep.scale, v);
        }
        if (t0.ep.base) v = fadd(t0.ep.base[t], fmul(t0.ep.coef, v));
        else if (t0.ep.zero_base) v = fadd(0.0f, fmul(t0.ep.coef, v));
        if (NT == 2) {
            float s1 = a1;
            if (t1.ep.potts) {
                if (t1.ep.norm) s1 = fmul(s1, s_nrm[1][li]);
                s1 = t1.ep.scale_vec ? fmul(t1.ep.scale_vec[k], s1) : fmul(t1.ep.scale, s1);
            }
            v = fadd(v, fmul(t1.ep.coef, s1));
        }
        return v;
    };
    const bool dense = s_dense;
    // The block shares its outer pixels with its neighbours.  With the labels at
    // compile time, or neither them nor the features, it walks all groups of its
    // pixels and skips those outside (kSkip), else (a pixel may be many blocks') from
    // the first element's group to the last's.  The whole filter, 640x480, by the
    // former and the latter: five features, 21 labels 269 us and 277, 40 labels 562
    // and 546; three features, 21 labels 221 and 231.
    const int ll = (ne - 1 + first) / L, last = ll * Q + (ne - 1 + first - ll * L) / 4;
    const int it0 = kSkip ? 0 : first / 4, it1 = kSkip ? np * Q : last + 1;
    for (int it = it0 + threadIdx.x; !dense && it < it1; it += blockDim.x) {
        const int li = it / Q, q = it - li * Q, e0 = li * L + 4 * q - first;
        if (kSkip && (e0 + 3 < 0 || e0 >= ne)) continue;
        const uint2 c = *reinterpret_cast<const uint2*>(bins + (long)(pf + li) * Lb + 4 * q);
        float a[NT][4];
#pragma unroll
        for (int h = 0; h < NT; h++) {
            const int2* ow = s_ow[h] + li * (h ? db : da);
            const float4* pl = reinterpret_cast<const float4*>(h ? t1.plane : t0.plane) + q;
            const float low = s_low[h][li];
            unsigned long long x = pack2(low, low), y = x;
            auto add = [&](int2 o) {
                const ulonglong2 r = *reinterpret_cast<const ulonglong2*>(pl + (long)o.x * Q);
                x = add_mul2(x, __int_as_float(o.y), r.x);
                y = add_mul2(y, __int_as_float(o.y), r.y);
            };
            if (h ? D1 : D0) {
#pragma unroll
                for (int j = 0; j <= (h ? D1 : D0); j++) add(ow[j]);
            } else {
                for (int j = 0; j < (h ? db : da); j++) add(ow[j]);
            }
            const float2 xl = unpack2(x), yl = unpack2(y);
            a[h][0] = xl.x;
            a[h][1] = xl.y;
            a[h][2] = yl.x;
            a[h][3] = yl.y;
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int e = e0 + i;
            if (4 * q + i >= L || e < 0 || e >= ne) continue;
            const unsigned ci = (i & 2 ? c.y : c.x) >> 16 * (i & 1) & 0xffffu;
            if (ci) s_hot[atomicAdd(&n_hot, 1)] = e | ci << 16;
            else s_val[e] = finish(a[0][i], a[NT - 1][i], li, 4 * q + i);
        }
    }
    __syncthreads();
    const int items = dense ? ne : n_hot;
    for (int n = threadIdx.x; n < items; n += blockDim.x) {
        const unsigned h = dense ? n | bin_of(n) << 16 : s_hot[n], c = h >> 16;
        const int e = h & 0xffff, f = e + first, li = f / L, k = f - li * L;
        const float a0 = ord_slice_sum<D0, kWide>(t0, s_ow[0] + li * da, k, c >> 8, c & 255, L);
        const float a1 = NT == 2 ? ord_slice_sum<D1, kWide>(t1, s_ow[1] + li * db, k, c >> 8, c & 255, L) : 0.0f;
        s_val[e] = finish(a0, a1, li, k);
    }
    __syncthreads();
    double g0 = 0.0, g1 = 0.0;
#pragma unroll
    for (int r = 0; r < kOsPer; r++) {
        const int e = r * kOsThreads + threadIdx.x;
        if (e < ne) {
            const float v = s_val[e];
            out[tb + e] = v;
            if (GAP) {
                const float tmp = fsub(ga[r], fadd(v, gf.su ? gf.su[tb + e] : 0.0f));
                g0 += (double)tmp * (double)gq[r];
                g1 += (double)tmp * (double)tmp;
            }
        }
    }
    if (GAP) gap_store(g0, g1, gf);
}

// The slice where a pixel's labels are too few to share its sums, or the
// elements too few to hide the phases above behind one another: one thread per
// element (kOsPer of them in turn; the same blocks, for the same partial sums),
// every vertex's float gathered (ord_slice_sum).
template <int D>
__device__ __forceinline__ float ord_slice_direct(const OrdSliceTerm& s, int i, int k, unsigned c, int L) {
    int2 ow[D + 1];
#pragma unroll
    for (int j = 0; j <= D; j++)
        ow[j] = make_int2(s.offset[(long)i * (D + 1) + j] + 1,
                          __float_as_int(fmul(s.bary[(long)i * (D + 1) + j], s.alpha)));
    return ord_slice_sum<D>(s, ow, k, c >> 8, c & 255, L);
}
template <bool GAP, int NT, int D0, int D1>
__global__ void __launch_bounds__(kOsThreads)
    ord_slice_direct_kernel(int N, int L, OrdSliceTerm t0, OrdSliceTerm t1, const unsigned short* __restrict__ bins,
                            float* out, GapFusion gf) {
    const int elems = slice_elems(L), Lb = ord_bin_row(L);
    const long NL = (long)N * L, tb = (long)blockIdx.x * elems;
    const int ne = (int)min((long)elems, NL - tb);
    double g0 = 0.0, g1 = 0.0;
    grid_release();
    grid_wait();
#pragma unroll
    for (int r = 0; r < kOsPer; r++) {
        const int e = r * kOsThreads + threadIdx.x;
        if (e < ne) {
            const long t = tb + e;
            const int i = (int)(t / L), k = (int)(t - (long)i * L);
            const unsigned c = bins[(long)i * Lb + k];
            float v = apply_epilogue(ord_slice_direct<D0>(t0, i, k, c, L), t, i, k, t0.ep);
            if (NT == 2) {
                float s1 = ord_slice_direct<D1>(t1, i, k, c, L);
                if (t1.ep.potts) {
                    if (t1.ep.norm) s1 = fmul(s1, t1.ep.norm[i]);
                    s1 = t1.ep.scale_vec ? fmul(t1.ep.scale_vec[k], s1) : fmul(t1.ep.scale, s1);
                }
                v = fadd(v, fmul(t1.ep.coef, s1));
            }
            out[t] = v;
            if (GAP) {
                const float al = fadd(gf.alpha[t], gf.u ? gf.u[t] : 0.0f);
                const float tmp = fsub(al, fadd(v, gf.su ? gf.su[t] : 0.0f));
                g0 += (double)tmp * (double)gf.Q[t];
                g1 += (double)tmp * (double)tmp;
            }
        }
    }
    if (GAP) gap_store(g0, g1, gf);
}

OrdSliceTerm slice_term(const Lattice& l, const SliceEpilogue& ep) {
    return OrdSliceTerm{l.offset.get(), l.bary.get(), l.ord_vals, l.ord_T.get() + (long)(l.d + 1) * (l.M + 1),
                        l.ord_plane.get(), l.d, 1.0f / (1.0f + std::pow(2.0f, (float)-l.d)), ep};
}

template <int NT>
void launch_slice(float* out, const unsigned short* bins, int L, const Lattice& a, const SliceEpilogue& ea,
                  const Lattice& b, const SliceEpilogue& eb, const GapFusion* gap, cudaStream_t st) {
    const long NL = (long)a.N * L;
    const OrdSliceTerm t0 = slice_term(a, ea), t1 = slice_term(b, eb);
    const int elems = slice_elems(L);
    // One thread per element, us: 640x480, five features, 4 labels, three calls
    // in flight 119 -> 106; the small LP (64x48, 21 labels, 6 steps) 6465 ->
    // 6252; from 2^17 values on it loses: the LP at 152x71 with 18 labels
    // 12430 -> 12640, at 200x120 with 21 labels 8340 -> 8800.
    const bool wide = L > kSliceElems;  // one term's only: a model has 64 labels at most
    require(!wide || (NT == 1 && !gap), DCRF_E_ARG, "ord_slice: too many labels");
    const bool known = !wide && (NT == 2 ? a.d == 2 && b.d == 5 : a.d == 2 || a.d == 5);
    if (known && (L < 8 || NL <= 1L << 17)) {
        auto direct = [&](auto kern) {
            launch_ord(NL, kern, ceil_div(NL, elems), kOsThreads, 0, st, a.N, L, t0, t1, bins, out,
                       gap ? *gap : GapFusion{});
        };
        auto by_d = [&](auto g) {
            constexpr bool GAP = decltype(g)::value;
            if constexpr (NT == 2) direct(ord_slice_direct_kernel<GAP, 2, 2, 5>);
            else if (a.d == 5) direct(ord_slice_direct_kernel<GAP, 1, 5, 5>);
            else direct(ord_slice_direct_kernel<GAP, 1, 2, 2>);
        };
        if (gap) by_d(std::true_type{});
        else by_d(std::false_type{});
        DCRF_LAUNCH_CHECK();
        return;
    }
    const int P = std::min(elems / L + 2, elems);  // pixels that a block touches at most
    auto bytes = [](int pixels, int d0, int d1) {
        return (sizeof(int2) + sizeof(float)) * pixels * (d0 + 1 + (NT == 2 ? d1 + 1 : 0)) + sizeof(float) * 4 * pixels;
    };
    const size_t smem = bytes(P, a.d, b.d);
    auto pick = [&](auto g) {
        constexpr bool GAP = decltype(g)::value;
        if constexpr (NT == 2) {
            return !known    ? ord_slice_kernel<GAP, NT, 0, 0, 0>
                   : L == 21 ? ord_slice_kernel<GAP, NT, 21, 2, 5>
                             : ord_slice_kernel<GAP, NT, 0, 2, 5>;
        } else {
            return wide       ? ord_slice_kernel<false, 1, -1, 0, 0>
                   : !known   ? ord_slice_kernel<GAP, NT, 0, 0, 0>
                   : a.d == 5 ? (L == 21 ? ord_slice_kernel<GAP, NT, 21, 5, 0> : ord_slice_kernel<GAP, NT, 0, 5, 0>)
                              : (L == 21 ? ord_slice_kernel<GAP, NT, 21, 2, 0> : ord_slice_kernel<GAP, NT, 0, 2, 0>);
        }
    };
    auto kern = gap ? pick(std::true_type{}) : pick(std::false_type{});
    // The opt-in is an attribute of the kernel that all threads share: always the
    // largest size there is (one label, two terms of 16 features: 53 KB).
    if (smem > 40 * 1024)
        DCRF_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)bytes(slice_elems(1), 16, 16)));
    launch_ord(NL, kern, ceil_div(NL, elems), kOsThreads, smem, st, a.N, L, P, t0, t1, bins, out, gap ? *gap : GapFusion{});
    DCRF_LAUNCH_CHECK();
}

}  // namespace

int ord_slice_grid(int N, int L) { return ceil_div((long)N * L, slice_elems(L)); }

size_t ordered_bins_size(long N, int L) { return (size_t)N * (ord_bin_row(L) + 2 * ord_words(L)); }

// The packed bins [N][ord_bin_row(L)], then the pixel masks [N][ord_words(L)].
static unsigned* bin_masks(const unsigned short* bins, long N, int L) {
    return reinterpret_cast<unsigned*>(const_cast<unsigned short*>(bins) + N * ord_bin_row(L));
}

void ordered_bins(unsigned short* bins, const float* Q, int N, int L, const float* qminmax, cudaStream_t st) {
    const long NL = (long)N * L;
    unsigned* pm = bin_masks(bins, N, L);
    if (L <= kBinTileMaxL) {
        launch_ord(NL, qminmax ? ord_bins_kernel<true> : ord_bins_kernel<false>, ceil_div(N, kBinTile * kOrdWarps),
                   kOrdThreads, sizeof(float) * kOrdWarps * ((kBinTile * L + 3) & ~3), st, N, L, Q, qminmax,
                   reinterpret_cast<uint4*>(bins), pm, (int)aligned16(Q));
    } else {  // a lattice's own call: a model, the only one to rescale, has 64 labels at most
        require(!qminmax, DCRF_E_ARG, "ordered_bins: too many labels to rescale");
        const int split = std::max(1, std::min((L + 31) / 32, (1 << 14) / N));
        launch_ord(NL, ord_bins_wide_kernel, dim3(ceil_div(N, kOrdWarps), split), kOrdThreads, 0, st, N, L, Q, bins, pm);
    }
    DCRF_LAUNCH_CHECK();
}

void Lattice::compute_ord(float* out, const float* Q, int L, const SliceEpilogue& ep) {
    require(L >= 1 && L <= kOrdMaxL, DCRF_E_ARG, "compute_ord: label count out of range");
    if (!ord_dense(L)) {
        try {
            unsigned short* bins = own(obins, ordered_bins_size(N, L));
            ordered_bins(bins, Q, N, L, nullptr, stream);
            ord_splat_blur(bins, L);
            ord_slice(out, bins, L, ep, nullptr);
            return;
        } catch (const Error& e) {  // the dense form's buffers beside the value buffers are fewer
            if (e.code != DCRF_E_NOMEM || (n_long && L > kOrdBlockMaxL)) throw;
            cudaGetLastError();
            give_back_quads();
        }
    }
    compute_ord_dense(out, Q, L, ep);
}

void Lattice::ord_splat_blur(const unsigned short* bins, int L) {
    require(L >= 1 && L <= kOrdMaxL, DCRF_E_ARG, "compute_ord: label count out of range");
    ensure_values((size_t)L * kOrdW);
    ensure_ord_totals();
    cudaStream_t st = stream;
    const int NW = ord_words(L), nblk = (L + 31) / 32, n_short = M - n_long;
    const int nc = std::min(4, ord_bin_row(L) / 8);
    float *src = va.get(), *dst = vb.get();
    unsigned *as = own(ord_a, (size_t)(M + 1) * NW), *ad = own(ord_b, (size_t)(M + 1) * NW);
    float* plane = own(ord_plane, (size_t)(M + 1) * ord_plane_row(L));
    const uint4* b4 = reinterpret_cast<const uint4*>(bins);
    const unsigned* pm = bin_masks(bins, N, L);
    if (n_long)
        launch_ord((long)N * L, NW == 4 ? ord_mask_kernel<4> : ord_mask_kernel<0>, n_long, 32 * kMaskWarps, 0, st, NW,
                       vorder.get(), seg_start.get(), seg.get(), pm, as);
    const long ht = (long)n_huge * nblk * kPairs, lt = (long)(n_long - n_huge) * nblk * kLongRounds;
    // Groups of lists or a thread per list and label: the latter where the lists have
    // few entries on average and are many; with many labels and vertices the group's
    // skipped quads win (noisy 640x480, 21 labels: an LP 101 ms by groups, 103 else).
    const bool few_lists = (long)N * (d + 1) < 8L * M && M >= 1 << 12 && (L <= 16 || M < 1 << 16);
    const long tasks = ht + lt + (few_lists ? ((long)n_short * L + 31) / 32 : (n_short + kGroup - 1) / kGroup);
    require(ht + lt < (1L << 30), DCRF_E_ARG, "compute_ord: too many labels");
    int bytes = std::max(n_long ? ord_ring_bytes(nc) + 2 * kUnitList : 0, few_lists ? 0 : ord_group_bytes(nc));
    bytes = (bytes + 15) & ~15;
    static_assert(kOrdWarps * (ord_ring_bytes(4) + 2 * kUnitList) <= (48 << 10) &&
                      kOrdWarps * ord_group_bytes(4) <= (48 << 10), "no opt-in to more shared memory");
    auto splat = few_lists ? (L == 21 ? ord_splat_kernel<3, 4, true> : ord_splat_kernel<0, 0, true>)
                           : (L == 21 ? ord_splat_kernel<3, 4, false> : ord_splat_kernel<0, 0, false>);
    launch_ord((long)N * L, splat, ceil_div(tasks, kOrdWarps), kOrdThreads, (size_t)bytes * kOrdWarps, st, M, n_long, n_huge,
                   (int)ht, (int)lt, L, NW, vorder.get(), seg_start.get(), seg.get(), b4, pm, as, ad, src, bytes);
    const bool few = NW == 1 && M >= 1 << 12;
    for (int j = 0; j <= d; j++) {
        const float* T = ord_T.get() + (long)j * (M + 1);
        auto pick = [&](auto last) {
            constexpr bool LAST = decltype(last)::value;
            return few       ? ord_blur_few_kernel<LAST>
                   : NW == 1 ? ord_blur_kernel<1, LAST>
                   : NW == 2 ? ord_blur_kernel<2, LAST>
                   : NW == 3 ? ord_blur_kernel<3, LAST>
                   : NW == 4 ? ord_blur_kernel<4, LAST>
                             : ord_blur_kernel<0, LAST>;
        };
        auto kern = j == d ? pick(std::true_type{}) : pick(std::false_type{});
        const int grid = few ? ceil_div((long)M * kQuads * L, kOrdBlurThreads)
                             : std::min(ceil_div(M, kOrdBlurThreads / 32), sm_count() * kOrdBlurBlocks);
        launch_ord((long)N * L, kern, grid, kOrdBlurThreads, 0, st, M, L, NW, nbr.get() + (long)j * M, T, T + M + 1,
                   reinterpret_cast<const float4*>(src), reinterpret_cast<float4*>(dst), as, ad, plane);
        std::swap(src, dst);
        std::swap(as, ad);
    }
    DCRF_LAUNCH_CHECK();
    ord_vals = src;
}

void Lattice::ord_slice_pair(float* out, const unsigned short* bins, int L, const Lattice& a, const SliceEpilogue& ea,
                             const Lattice& b, const SliceEpilogue& eb, const GapFusion* gap) {
    require(a.ord_vals && b.ord_vals, DCRF_E_STATE, "ord_slice_pair: no ord_splat_blur before it");
    require(a.N == b.N, DCRF_E_ARG, "ord_slice_pair: lattices over different pixel counts");
    launch_slice<2>(out, bins, L, a, ea, b, eb, gap, a.stream);
}

void Lattice::ord_slice(float* out, const unsigned short* bins, int L, const SliceEpilogue& ep, const GapFusion* gap) {
    require(ord_vals, DCRF_E_STATE, "ord_slice: no ord_splat_blur before it");
    launch_slice<1>(out, bins, L, *this, ep, *this, ep, gap, stream);
}

namespace {

__global__ void fill_int_kernel(long n, int v, int* __restrict__ x) {
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) x[t] = v;
}

}  // namespace

namespace {

__global__ void pair_bins_kernel(long n, const float* __restrict__ Q, float2* __restrict__ bins) {
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    bins[t] = ord_bin_pair(Q[t]);
}

// The same, four elements per thread with 16-byte loads and stores (Q and
// bins 16-byte aligned; n4 = n / 4 quads, the tail by pair_bins_kernel).
__global__ void pair_bins4_kernel(long n4, const float4* __restrict__ Q, float4* __restrict__ bins) {
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n4) return;
    const float4 q = Q[t];
    const float2 a = ord_bin_pair(q.x), b = ord_bin_pair(q.y), c = ord_bin_pair(q.z), d = ord_bin_pair(q.w);
    bins[2 * t] = make_float4(a.x, a.y, b.x, b.y);
    bins[2 * t + 1] = make_float4(c.x, c.y, d.x, d.y);
}

// (c_lower, c_upper) of Q [n] as floats, for the restricted filter: four per
// thread where the pointers allow.
void pair_bins(float2* bins, const float* Q, long n, cudaStream_t st) {
    if (aligned16(Q) && aligned16(bins)) {
        const long n4 = n / 4;
        if (n4) launch(pair_bins4_kernel, ceil_div(n4, kTB), kTB, 0, st, n4, reinterpret_cast<const float4*>(Q),
                       reinterpret_cast<float4*>(bins));
        if (n > 4 * n4) launch(pair_bins_kernel, 1, kTB, 0, st, n - 4 * n4, Q + 4 * n4, bins + 4 * n4);
    } else {
        launch(pair_bins_kernel, ceil_div(n, kTB), kTB, 0, st, n, Q, bins);
    }
}

// ---------------------------------------------------------------------------
// The dense form: every bin of every label, nothing skipped (ord_dense); a
// vertex row holds 20 bins x L labels, bin-major ([v][bin][label]; bins [0,10)
// lower, [10,20) upper) so that the slice's per-label bin reads coalesce.  Where no
// list is long its kernels touch little more than the quads that exist and leave
// most of the chip's registers and all of its shared memory to other streams.

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

// Its long lists, by blocks.  The 20 x L bin sums of a
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
constexpr int kHugeLabels = 12;         // labels per block for the lists over kHugeList
constexpr int kOE = 32;                 // entries per chunk
constexpr int kODX = 4;                 // bins are copied kODX chunks ahead of use, pixel ids 2 kODX
constexpr int kOXS = kODX + 1;          // bin ring slots (chunks c .. c+kODX)
constexpr int kOPS = 2 * kODX + 1;      // pixel / weight ring slots (chunks c .. c+2 kODX)
constexpr int kORow = 2 * kOE + 4;      // floats per ring row: 17 x 16 bytes
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
    ord_dense_long_kernel(int L, int kb, int kblocks, const int* __restrict__ order,
                           const int* __restrict__ seg_start, const int2* __restrict__ seg,
                           const float2* __restrict__ bins, float* __restrict__ vals) {
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

// Splat of the short lists (order: those past the long ones; null: every list), one
// thread per (vertex, label), both passes in registers: lower bin 0
// and upper bin 9 take every entry, the other 18 bins an FMA with a mask of
// exactly 0 or 1 (fma(1, w, acc) is acc + w rounded once).  Also clears the
// absent neighbour's row in both buffers.
__global__ void ord_dense_splat_kernel(int n_short, int L, const int* __restrict__ order,
                                       const int* __restrict__ seg_start, const int2* __restrict__ seg,
                                       const float2* __restrict__ bins, float* __restrict__ vals,
                                       float* __restrict__ other) {
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    for (long z = t; z < (long)kOrdW * L; z += (long)gridDim.x * blockDim.x) vals[z] = other[z] = 0.0f;
    if (t >= (long)n_short * L) return;
    const int u = (int)(t / L), k = (int)(t - (long)u * L), v = order ? order[u] : u;
    const int s0 = seg_start[v], s1 = seg_start[v + 1];
    float lo[kRes], up[kRes];
#pragma unroll
    for (int b = 0; b < kRes; b++) lo[b] = up[b] = 0.0f;
#pragma unroll 2
    for (int s = s0; s < s1; s++) {
        const int2 en = seg[s];
        const float2 x = bins[(long)en.x * L + k];
        const float w = entry_w(en);
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

// One axis, one thread per four values.  R4: a row's float4 at compile time (0: row4r).
template <int R4>
__global__ void ord_dense_blur_kernel(int M, int row4r, const int2* __restrict__ nbr, const float4* __restrict__ src,
                                      float4* __restrict__ dst) {
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

// Slice, one thread per (pixel, label): the lower pass, then the upper.
template <int DC, int LC>
__global__ void __launch_bounds__(kTB, 8)
    ord_dense_slice_kernel(int N, int Lrt, int drt, const int* __restrict__ offset, const float* __restrict__ bary,
                           const float* __restrict__ vals, const float2* __restrict__ bins, float alpha, float* out,
                           SliceEpilogue ep) {
    const int L = LC ? LC : Lrt, d = DC ? DC : drt;
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long)N * L) return;
    const int i = (int)(t / L), k = (int)(t - (long)i * L), d1 = d + 1;
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
    out[t] = apply_epilogue(acc, t, i, k, ep);
}
}  // namespace

void Lattice::ensure_aux() {
    if (aux) return;
    int lo = 0, hi = 0;
    DCRF_CUDA(cudaDeviceGetStreamPriorityRange(&lo, &hi));
    DCRF_CUDA(cudaEventCreateWithFlags(&ev_fork, cudaEventDisableTiming));
    DCRF_CUDA(cudaEventCreateWithFlags(&ev_join, cudaEventDisableTiming));
    DCRF_CUDA(cudaStreamCreateWithPriority(&aux, cudaStreamNonBlocking, hi));
}

Lattice::~Lattice() {
    if (aux) {
        cudaStreamSynchronize(aux);
        cudaStreamDestroy(aux);
    }
    if (ev_join) cudaEventDestroy(ev_join);
    if (ev_fork) cudaEventDestroy(ev_fork);
}

// Whether a single filter takes the dense form (the LP's fused slice needs the
// quad form).  The lines lie where the two cross on a solver's kind of values
// (softmax of normal logits); one call after the other, us, quad form -> dense.
//   No long list, two features at most: from 2^19 (pixel, label) values or 2^18
//   pixels on; from 20 labels on where there are pixels to fill the chip, and
//   above 28 labels, whose masks are read in a loop.  640x480 with 3 labels 70 ->
//   51, 21 labels 205 -> 207, and 215 -> 178 with three calls in flight; 160x120
//   with 22 labels 41.5 -> 39.9, 97x83 with 32 49 -> 36; below the lines 320x240
//   with 2 labels 25 -> 34, 97x83 with 21 30 -> 37.
//   Else the quad form wins where long lists leave most quads empty (five
//   features, 640x480, 21 labels 272 -> 362), and loses with few labels: a list's
//   sums fill few lanes (640x480: 2 labels 131 -> 107, 8 192 -> 182, 12 232 ->
//   231, 16 259 -> 289; 320x240, whose splat does not fill the chip: 12 labels
//   123 -> 112, 20 146 -> 142, 26 180 -> 207; smaller ones win throughout), and its
//   masks cost by the vertex whatever the labels: a noisy image 640x480, 650
//   thousand vertices, 2 labels 496 -> 409, 4 929 -> 709, 21 3949 -> 3659, 32 5159
//   -> 5482; 320x240, 178 thousand, 4 labels 255 -> 215, 20 902 -> 916; 160x120, 52
//   thousand, 4 labels 64 -> 70.
// On evenly spread values, where all quads exist, the quad form loses everywhere
// (five features, 640x480, 21 labels 379 -> 350): a single filter of those is
// slower than the dense form would be.
bool Lattice::ord_dense(int L) const {
    if (n_long && L > kOrdBlockMaxL) return false;
    if (d <= 2 && n_long == 0)
        return (long)N * L > 1L << 19 || N > 1 << 18 || L > 28 || (L >= 20 && N >= 1 << 14);
    const bool long_lists = (long)N * (d + 1) >= 32L * M;  // on average
    return L <= (!long_lists ? 0 : N > 1 << 18 ? 12 : N > 1 << 16 ? 20 : 0) || ord_many(L);
}

// ... for the number of its vertices: from 60 thousand on for one label, eight more
// with each doubling.
bool Lattice::ord_many(int L) const {
    return (d > 2 || n_long) && L <= kOrdBlockMaxL && L <= 8.0 * std::log2((double)M) - 127.0;
}

void Lattice::compute_ord_dense(float* out, const float* Q, int L, const SliceEpilogue& ep) {
    const size_t row = (size_t)L * kOrdW;
    ensure_values(row);
    cudaStream_t st = stream;
    const long NL = (long)N * L;
    float2* bins = own(r_ebins, (size_t)NL);
    pair_bins(bins, Q, NL, st);
    float *src = va.get(), *dst = vb.get();
    const int n_short = M - n_long;
    auto long_lists = [&](int G, int kb, int first, int count, cudaStream_t ls) {
        if (count <= 0) return;
        const int kblocks = (L + kb - 1) / kb;
        const size_t smem = ord_block_smem(kb);
        auto kern = G == 10 ? ord_dense_long_kernel<10>
                  : G == 5  ? ord_dense_long_kernel<5>
                  : G == 3  ? ord_dense_long_kernel<3>
                  : G == 2  ? ord_dense_long_kernel<2>
                            : ord_dense_long_kernel<1>;
        // an attribute of the kernel that all threads share: always its largest size
        if (smem > 48 * 1024)
            DCRF_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)ord_block_smem(kOrdBlockMaxL)));
        launch(kern, count * kblocks, (kb * G + 31) / 32 * 32, smem, ls, L, kb, kblocks,
               (const int*)vorder.get() + first, (const int*)seg_start.get(), (const int2*)seg.get(),
               (const float2*)bins, src);
    };
    // The very long lists set the length of their kernel and leave most SMs
    // idle: on a stream of their own, joined before the blur, beside the others
    // (other rows of src).
    if (n_huge) {
        ensure_aux();
        DCRF_CUDA(cudaEventRecord(ev_fork, st));
        DCRF_CUDA(cudaStreamWaitEvent(aux, ev_fork, 0));
        long_lists(10, std::min(L, kHugeLabels), 0, n_huge, aux);
        DCRF_CUDA(cudaEventRecord(ev_join, aux));
    }
    if (n_long > n_huge) long_lists(ord_groups_cheapest(L), L, n_huge, n_long - n_huge, st);
    launch(ord_dense_splat_kernel, std::max(1, ceil_div((long)n_short * L, kTB)), kTB, 0, st, n_short, L,
           n_long ? (const int*)vorder.get() + n_long : nullptr, (const int*)seg_start.get(), (const int2*)seg.get(),
           (const float2*)bins, src, dst);
    if (n_huge) DCRF_CUDA(cudaStreamWaitEvent(st, ev_join, 0));
    const int row4 = (int)(row / 4);
    for (int j = 0; j <= d; j++) {
        launch(row4 == 105 ? ord_dense_blur_kernel<105> : ord_dense_blur_kernel<0>, ceil_div((long)M * row4, kTB), kTB,
               0, st, M, row4, (const int2*)(nbr.get() + (long)j * M), reinterpret_cast<const float4*>(src),
               reinterpret_cast<float4*>(dst));
        std::swap(src, dst);
    }
    const float alpha = 1.0f / (1.0f + std::pow(2.0f, (float)-d));
    auto slice = d == 2 ? (L == 21 ? ord_dense_slice_kernel<2, 21> : ord_dense_slice_kernel<2, 0>)
                        : ord_dense_slice_kernel<0, 0>;
    launch(slice, ceil_div(NL, kTB), kTB, 0, st, N, L, d, (const int*)offset.get(), (const float*)bary.get(),
           (const float*)src, (const float2*)bins, alpha, out, ep);
    DCRF_LAUNCH_CHECK();
    ord_vals = nullptr;  // the buffers hold no quads
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
    if (store) r_L = 0;  // until this call has stored its splat
    const long row = (long)L * kOrdW, cells = (long)(M + 1) * row;
    float* stored = own(r_stored, (size_t)cells);
    float* a = own(r_a, (size_t)cells);
    float* b = own(r_b, (size_t)cells);
    unsigned char* active = own(r_active, (size_t)std::max(M, 1));
    int* pos = own(r_pos, (size_t)N);
    float2* rb = own(r_bins, (size_t)std::max<long>((long)nP * L, 1));
    launch(fill_int_kernel, ceil_div(N, kTB), kTB, 0, st, (long)N, -1, pos);
    if (nP) {
        launch(scatter_pos_kernel, ceil_div(nP, kTB), kTB, 0, st, nP, pI, pos);
        pair_bins(rb, rQ, (long)nP * L, st);
    }
    const float2* eb = nullptr;
    if (store) {
        float2* e = own(r_ebins, (size_t)N * L);
        pair_bins(e, Q, (long)N * L, st);
        eb = e;
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
