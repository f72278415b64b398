// Device-wide integer primitives used to build the lattice deterministically:
// an exclusive prefix sum and a stable LSD radix sort of (key, value) pairs.
#pragma once
#include "common.cuh"

namespace dcrf {

// Scratch owned by the caller so repeated builds do not reallocate.
struct ScanScratch {
    DevBuf<int> block_sums;
};

// out[i] = sum_{j<i} in[i]; in may alias out.  If d_total is non-null the
// grand total is written there (device pointer).  n < 2^31.
void exclusive_scan(const int* in, int* out, int n, int* d_total, ScanScratch& s,
                    cudaStream_t st);

// ranks[e] = number of e' < e with table[slot[e']] == e' (exclusive scan of the
// first-occurrence flags); their total to d_total.
void first_flags_scan(const int* slot, const int* table, int n, int* ranks, int* d_total, ScanScratch& s,
                      cudaStream_t st);

struct SortScratch {
    DevBuf<int> keys_alt, vals_alt, hist;
    ScanScratch scan;
};

// Stable sort of keys[0..n) (0 <= key < 2^key_bits) carrying vals; the
// result is left in keys/vals.  Equal keys keep their input order, so a
// sort of (vertex id, entry index) pairs yields per-vertex entry lists in
// increasing entry order.
void radix_sort_pairs(int* keys, int* vals, int n, int key_bits, SortScratch& s, cudaStream_t st);
// The same with the values 0 .. n-1 and the keys left as they are: the sorted
// keys and indexes are returned in buffers of the scratch or in kbuf / vbuf [n].
void radix_sort_index(const int* keys, int n, int key_bits, int* kbuf, int* vbuf, const int** keys_out,
                      const int** vals_out, SortScratch& s, cudaStream_t st);

}  // namespace dcrf
