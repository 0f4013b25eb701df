// 1-bit ROSA match by the latest position of every context: the idx of RosaSam::push (src/rosa.rs:100-176) for streams
// whose keys are spread evenly.
//
// What a step needs (rosa_match.cuh says why) is the position r < t whose key history agrees with the query history of
// step t over the most steps, the latest one of equals.  A warp walks along a stream 32 steps (a row) at a time and keeps
// the latest position of every context of up to DEPTH bits that lies before the row; inside the row the positions that
// agree are bit masks, refined by one bit of the histories after the other.  The longest of the contexts that was met is
// the answer up to DEPTH - 1 bits; the positions that agree in DEPTH bits or more form a chain from the latest to the
// earliest, which is walked.
//
// Positions are held as r + 1, so 0 is none.  Histories are filled up with zeros before the first step.  A position
// that agrees in d bits has at least d steps behind it only if r + 1 >= d, so a context of d bits counts only if its
// latest position has; if that one has not, none of the context has.
#pragma once
#include <stdint.h>

#include "rosa_context.cuh"

namespace ullis {
namespace heads {

// Contexts of 11, 7 and 3 bits are stored: eight that lie side by side answer for the three lengths below as well (the
// later of two contexts of d bits is the latest of their common d - 1 bits).  11 bits: of 2048 steps one position per
// context; the chains of the model's streams (default model, gain 1 + N(0, 0.02)) are 3.3 positions long for the longest
// of 32 steps, with 10 bits 5.4, with 12 bits 2.1 but twice the shared memory.
constexpr uint32_t DEPTH = 11;
constexpr uint32_t LATEST_11 = 2048, LATEST_7 = 128, LATEST_3 = 8;   // u16, u32 and u32 each, eight side by side aligned to their size

RC_HD uint32_t later(uint32_t a, uint32_t b) { return a > b ? a : b; }

// p0 .. p3: the latest position + 1 of the query's contexts of d .. d - 3 bits (0: none).  The longest that counts, as
// bits << 16 | position + 1, 0 if there is none.
RC_HD uint32_t deepest(uint32_t p0, uint32_t p1, uint32_t p2, uint32_t p3, uint32_t d) {
    uint32_t found = d > 3u && p3 >= d - 3u ? (d - 3u) << 16 | p3 : 0u;
    if (p2 >= d - 2u) found = (d - 2u) << 16 | p2;
    if (p1 >= d - 1u) found = (d - 1u) << 16 | p1;
    if (p0 >= d) found = d << 16 | p0;
    return found;
}
// The query whose window is wq among the contexts of 11 bits ...
RC_HD uint32_t probe_11(const uint16_t* table, uint32_t wq) {
    const uint32_t ctx = wq >> 21;
#if defined(__CUDA_ARCH__)
    const uint4 x = *reinterpret_cast<const uint4*>(table + (ctx & ~7u));
    const uint32_t a = ctx & 4u ? x.z : x.x, b = ctx & 4u ? x.w : x.y, pair = ctx & 2u ? b : a;
    const uint32_t quad = __vmaxu2(a, b), all = __vmaxu2(__vmaxu2(x.x, x.y), __vmaxu2(x.z, x.w));
    const uint32_t own = __funnelshift_r(pair, 0u, ctx << 4);   // modulo 32: the half of an even or odd context
    const uint32_t both = __vmaxu2(__byte_perm(pair, quad, 0x5410u), __byte_perm(pair, quad, 0x7632u));
    return deepest(own & 0xFFFFu, both & 0xFFFFu, both >> 16, later(all & 0xFFFFu, all >> 16), DEPTH);
#else
    auto among = [&](uint32_t n) {
        uint32_t p = 0;
        for (uint32_t i = ctx / n * n; i < ctx / n * n + n; ++i) p = later(p, table[i]);
        return p;
    };
    return deepest(among(1), among(2), among(4), among(8), DEPTH);
#endif
}
// ... and of d = 7 or 3 bits.
RC_HD uint32_t probe(const uint32_t* table, uint32_t wq, uint32_t d) {
    const uint32_t ctx = wq >> (32u - d);
#if defined(__CUDA_ARCH__)
    const uint4 u = *reinterpret_cast<const uint4*>(table + (ctx & ~7u)), w = *reinterpret_cast<const uint4*>(table + (ctx | 4u) - (ctx & 3u));
    const bool upper = ctx & 4u;
    const uint32_t a = upper ? w.x : u.x, b = upper ? w.y : u.y, c = upper ? w.z : u.z, e = upper ? w.w : u.w;
    const uint32_t even = ctx & 2u ? c : a, odd = ctx & 2u ? e : b, quad = later(later(a, b), later(c, e));
    const uint32_t all = later(later(later(u.x, u.y), later(u.z, u.w)), later(later(w.x, w.y), later(w.z, w.w)));
    return deepest(ctx & 1u ? odd : even, later(even, odd), quad, all, d);
#else
    auto among = [&](uint32_t n) {
        uint32_t p = 0;
        for (uint32_t i = ctx / n * n; i < ctx / n * n + n; ++i) p = later(p, table[i]);
        return p;
    };
    return deepest(among(1), among(2), among(4), among(8), d);
#endif
}

// Bit d of a window, counted from 1 at the top, in all bits.  One shift serves the bits of several bytes: a byte permutation
// repeats the sign of a byte.
RC_HD uint32_t spread(uint32_t w, uint32_t d) {
#if defined(__CUDA_ARCH__)
    uint32_t all;
    asm("prmt.b32 %0, %1, 0, %2;" : "=r"(all) : "r"(w << ((d - 1u) & 7u)), "r"(0xBBBBu - 0x1111u * ((d - 1u) >> 3)));
    return all;
#else
    return 0u - (w >> (32u - d) & 1u);
#endif
}
// Of the lanes below this one those whose keys agree longest with the query history wq, up to DEPTH bits (0: none agrees in
// one).  before, now: the key words of the row before and of the row.  FIRST: it is the first of its stream, where lane r has
// only r + 1 steps behind it.
template <bool FIRST>
RC_HD uint32_t agreeing(uint32_t before, uint32_t now, uint32_t below, uint32_t wq) {
    uint32_t lanes = below, best = 0;
#if defined(__CUDACC__)
#pragma unroll
#endif
    for (uint32_t d = 1; d <= DEPTH; ++d) {
        // bit j: the key d - 1 steps before position j of the row
#if defined(__CUDA_ARCH__)
        const uint32_t bits = __funnelshift_l(before, now, d - 1u);
#else
        const uint32_t bits = d > 1u ? now << (d - 1u) | before >> (33u - d) : now;
#endif
        lanes &= ~(bits ^ spread(wq, d));
        const uint32_t full = FIRST ? lanes & 0xFFFFFFFFu << (d - 1u) : lanes;
        if (full) best = full;
    }
    return best;
}
RC_HD uint32_t latest(uint32_t row, uint32_t lanes) { return 32u * row + 32u - context::leading(lanes); }   // r + 1, lanes != 0

// The window that ends with position r1 - 1, r1 < 32 * words; W as in rosa_context.cuh.
RC_HD uint32_t window_before(const uint32_t* W, uint32_t r1) {
    const uint32_t lo = W[r1 >> 5], sh = r1 & 31u;
#if defined(__CUDA_ARCH__)
    return __funnelshift_r(lo, W[(r1 >> 5) + 1u], sh);
#else
    return sh ? lo >> sh | W[(r1 >> 5) + 1u] << (32u - sh) : lo;
#endif
}

// The positions of a word that end a run of DEPTH ones inside it.
RC_HD uint32_t ends_of_runs(uint32_t x) {
    x &= x << 1;
    x &= x << 2;
    x &= x << 4;
    return x & x << 3;   // 8 and 3
}
// Whether the walks of rows with queries in the one context of such a run, `rows` of them, come to more than `most` positions if
// `keys` positions are in it: on average half of those lie before a row.
RC_HD bool walks_too_long(uint32_t keys, uint32_t rows, uint32_t most) { return keys * rows > 2u * most; }

// A stream of `words` rows in pieces of equal length, the last one shorter; of the pieces that are wanted as many as have a row
// (a piece without any would put in all keys of the stream and answer nothing: 33 steps in four pieces have two such).
constexpr uint32_t rows_of_piece(uint32_t words, uint32_t pieces) { return (words + pieces - 1u) / pieces; }
constexpr uint32_t pieces_with_rows(uint32_t words, uint32_t wanted) { return rows_of_piece(words, rows_of_piece(words, wanted)); }

}  // namespace heads
}  // namespace ullis
