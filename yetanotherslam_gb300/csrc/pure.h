// pure.h — arithmetic of calls and kernels that needs no GPU, in a header of
// its own so that host tests compile the same lines.
#pragma once

#include <stddef.h>

#ifdef __CUDACC__
#define YAS_PURE __host__ __device__ __forceinline__
#define YAS_UNROLL _Pragma("unroll")
#define YAS_NO_UNROLL _Pragma("unroll 1")
#else
#define YAS_PURE inline
#define YAS_UNROLL
#define YAS_NO_UNROLL
#endif

namespace yas {

// Bytes from the first to the last byte of an image of `rows` rows of
// `row_bytes`, `pitch` bytes apart: the padding behind the last row is not the
// image's, and need not be there.
inline size_t image_bytes(size_t row_bytes, size_t pitch, int rows) { return pitch * (size_t)(rows - 1) + row_bytes; }

// 4.685 sd, the FP64 product rounded once to FP32.  (An FP32 product with 4.685 to
// 48 bits, its parts summed, is a last place off for one sd in 2800, on the wrong
// side of a near tie, and is not a number for an infinite one.)
YAS_PURE float huber_scaled(float sd) { return (float)(4.685 * (double)sd); }

// A cell of a raycast's block grid, its epoch taken off: a pool index below
// kGridAsk; kGridAsk where the index does not fit (the hash table has it); above,
// no allocated block.
constexpr unsigned kGridAsk = 0xffffffu;

// Pool index of the block of each corner of a 2x2x2 voxel cell that straddles the
// block faces of the axes in `across` (1 x, 2 y, 4 z; not 0): corner c lies in
// neighbour c & across of the block b that holds corner 0.  An index at or above
// the returned limit is that of no allocated block.  inner: the grid holds b and
// its upper neighbours, whose cells word(c) reads (c's axes outside `across` are
// without effect); they are read side by side.  Otherwise, or when an index does
// not fit the grid, b's own among them, lookup(d) finds neighbour d, or -1, one by
// one.
template <class Word, class Lookup>
YAS_PURE unsigned corner_blocks(unsigned across, int b, bool inner, Word word, Lookup lookup, unsigned q[8]) {
    bool ask = !inner || (unsigned)b >= kGridAsk;
    q[0] = (unsigned)b;
    if (!ask) {
        YAS_UNROLL
        for (unsigned c = 1; c < 8; ++c) {
            q[c] = word(c);
            ask = ask || q[c] == kGridAsk;
        }
    }
    if (!ask) return kGridAsk;
    YAS_UNROLL
    for (unsigned c = 1; c < 8; ++c) q[c] = (unsigned)b;
    YAS_NO_UNROLL
    for (unsigned d = across; d != 0u; d = (d - 1u) & across) {
        const int e = lookup(d);
        YAS_UNROLL
        for (unsigned c = 1; c < 8; ++c) q[c] = (c & across) == d ? (unsigned)e : q[c];
    }
    return 0x80000000u;
}

}  // namespace yas
