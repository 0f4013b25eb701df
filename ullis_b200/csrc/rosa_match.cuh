// 1-bit ROSA match by sets of lags: the second way to the idx of RosaSam::push (src/rosa.rs:100-176), without an
// automaton and without a chain of steps that has to run from the first one.
//
// What push computes.  The query state of the automaton is the class of the longest suffix of q[0..t] that occurs in
// the keys so far, the `last` it reads is the latest end of an occurrence, and idx is the v bit after it:
//
//     L(t)   = the longest L with q[t-L+1..t] = k[r-L+1..r] for some r < t          (0: no match, idx = 0)
//     d(t)   = t - r for the latest such r, i.e. the smallest lag d with q[j] = k[j-d] for all j in (t-L, t]
//     idx(t) = v[t - d(t) + 1]
//
// (the climb of src/rosa.rs:121-127 never leaves the state the transition reached: it compares link lengths with a
// match length that is never below the true one).  With X(j) = { d : 1 <= d <= j, q[j] = k[j-d] } as a bit set over
// the lags, L(t) is the longest window (s, t] whose X(j) have a lag in common, and its start only moves forward:
// L(t) <= L(t-1) + 1.  So one warp keeps the intersection E of the current window in registers (32 * NW words, NW per
// lane) and extends it by one AND per step; when E runs empty the window loses its oldest steps.  Intersections cannot
// be undone, so the window is kept as a queue out of two stacks: `front` holds the suffix intersections
// S(i) = X(i) & ... & X(mid) for i = s..mid, `back` the intersection of the steps after mid.  Dropping the oldest
// step is one load (S(s+1) & back); when the front is used up it is rebuilt from the current step downwards until the
// intersection is empty, which is at the same time the search for the next window.  Every step enters and leaves each
// stack once: three set operations per step on average, whatever the streams look like.
//
// The window at any step can be found from scratch by that same rebuild, so a stream is cut into pieces of steps that
// know nothing of one another: there is no serial chain over the stream.
//
// The front is kept in a ring of the oldest sets of the window.  A longer window (they reach the whole stream where a
// bit hardly ever changes) leaves every `gap`-th set in global memory on the way down, and the ring is refilled from
// the next of those when it is used up.
//
// The code is written for a warp as one value per lane (`lv`), so that the same source runs host-compiled with a lane
// array in the tests.
#pragma once
#include <stdint.h>

#if defined(__CUDACC__)
#define RM_HD __device__ __forceinline__
#define RM_BOTH __host__ __device__ __forceinline__
#else
#define RM_HD inline
#define RM_BOTH inline
#endif

namespace ullis {
namespace match {

// ---- one value per lane
#if defined(__CUDACC__)
typedef uint32_t lv;
RM_HD lv lv_all(uint32_t x) { return x; }
RM_HD lv lv_load(const uint32_t* p) { return p[threadIdx.x & 31u]; }
RM_HD void lv_store(uint32_t* p, lv x) { p[threadIdx.x & 31u] = x; }
RM_HD lv lv_funnel(lv lo, lv hi, uint32_t sh) { return __funnelshift_r(lo, hi, sh); }
RM_HD lv lv_xor(lv a, uint32_t m) { return a ^ m; }
RM_HD uint32_t lv_ballot(lv x) { return __ballot_sync(0xFFFFFFFFu, x != 0u); }
RM_HD uint32_t lv_from(lv x, uint32_t lane) { return __shfl_sync(0xFFFFFFFFu, x, (int)lane); }
RM_HD uint32_t& lv_at(lv& x, uint32_t) { return x; }
RM_HD uint32_t ctz32(uint32_t x) { return (uint32_t)__ffs((int)x) - 1u; }
RM_HD uint32_t funnel32(uint32_t lo, uint32_t hi, uint32_t sh) { return __funnelshift_r(lo, hi, sh); }
RM_HD uint32_t brev32(uint32_t x) { return __brev(x); }
RM_HD void warp_sync() { __syncwarp(); }
#define RM_LANES(l) for (uint32_t l = threadIdx.x & 31u, rm_once = 1u; rm_once; rm_once = 0u)
#else
struct lv { uint32_t v[32]; };
inline lv operator&(lv a, const lv& b) { for (int i = 0; i < 32; ++i) a.v[i] &= b.v[i]; return a; }
inline lv operator|(lv a, const lv& b) { for (int i = 0; i < 32; ++i) a.v[i] |= b.v[i]; return a; }
inline lv lv_all(uint32_t x) { lv a; for (int i = 0; i < 32; ++i) a.v[i] = x; return a; }
inline lv lv_load(const uint32_t* p) { lv a; for (int i = 0; i < 32; ++i) a.v[i] = p[i]; return a; }
inline void lv_store(uint32_t* p, const lv& x) { for (int i = 0; i < 32; ++i) p[i] = x.v[i]; }
inline uint32_t funnel32(uint32_t lo, uint32_t hi, uint32_t sh) { return (sh &= 31u) ? lo >> sh | hi << (32u - sh) : lo; }
inline lv lv_funnel(const lv& lo, const lv& hi, uint32_t sh) { lv a; for (int i = 0; i < 32; ++i) a.v[i] = funnel32(lo.v[i], hi.v[i], sh); return a; }
inline lv lv_xor(lv a, uint32_t m) { for (int i = 0; i < 32; ++i) a.v[i] ^= m; return a; }
inline uint32_t lv_ballot(const lv& x) { uint32_t b = 0; for (int i = 0; i < 32; ++i) b |= (uint32_t)(x.v[i] != 0u) << i; return b; }
inline uint32_t lv_from(const lv& x, uint32_t lane) { return x.v[lane]; }
inline uint32_t& lv_at(lv& x, uint32_t l) { return x.v[l]; }
inline uint32_t ctz32(uint32_t x) { return (uint32_t)__builtin_ctz(x); }
inline uint32_t brev32(uint32_t x) { uint32_t r = 0; for (int i = 0; i < 32; ++i) r |= (x >> i & 1u) << (31 - i); return r; }
inline void warp_sync() {}
#define RM_LANES(l) for (uint32_t l = 0; l < 32u; ++l)
#endif

// Words of shared memory one warp needs for pieces whose last step lies below 1024 * nw_max, with a ring of
// ring_words words.
struct Layout {
    uint32_t r1, r0, qs, ks, ring, total;
    RM_BOTH Layout(uint32_t nw_max, uint32_t ring_words) {
        const uint32_t rev = 64u * nw_max + 32u, fwd = 32u * nw_max + 32u;   // both with room for reads past the end
        r1 = 0; r0 = rev; qs = 2u * rev; ks = qs + fwd; ring = ks + fwd; total = ring + ring_words;
    }
};

// Sets that a warp may leave in global memory for streams of T steps, and the distance between two of them.
constexpr uint32_t CHECKPOINTS = 64;
RM_BOTH uint32_t checkpoint_gap(uint32_t T) {
    uint32_t g = 16u;
    while (g * CHECKPOINTS < T) g <<= 1;
    return g;
}

// The steps [t0, t1) of one stream (t0 a multiple of 32, t1 <= T, t1 <= 1024 * NW); all lanes of a
// warp call it together.  mem: Layout::total words of shared memory; kept: CHECKPOINTS * 32 * NW words of the warp's own.
template <int NW>
RM_HD void piece(uint32_t* mem, const Layout& L, uint32_t ring_words, uint32_t* kept, uint32_t gap, const uint32_t* __restrict__ qw,
                 const uint32_t* __restrict__ kw, const uint32_t* __restrict__ vw, uint32_t* __restrict__ idx,
                 uint32_t t0, uint32_t t1) {
    uint32_t* const R1 = mem + L.r1;     // bit P-1-i = [k_i = 1], zero from bit P on: k backwards
    uint32_t* const R0 = mem + L.r0;     // bit P-1-i = [k_i = 0], zero from bit P on
    uint32_t* const qs = mem + L.qs;
    uint32_t* const ks = mem + L.ks;
    uint32_t* const ring = mem + L.ring;
    const uint32_t words = (t1 + 31u) / 32u;          // <= 32 * NW
    const uint32_t P = words * 32u;
    const uint32_t D = ring_words / (32u * NW);       // sets in the ring, a power of two
    warp_sync();                                       // the lanes may still be reading the piece before this one
    RM_LANES(l) {
        for (uint32_t w = l; w < words + 32u * NW + 1u; w += 32u) {
            const uint32_t x = w < words ? brev32(kw[words - 1u - w]) : 0u;
            R1[w] = x;
            R0[w] = w < words ? ~x : 0u;
        }
        for (uint32_t w = l; w < words + 1u; w += 32u) {
            qs[w] = w < words ? qw[w] : 0u;
            ks[w] = w < words ? kw[w] : 0u;
        }
    }
    warp_sync();

    // X(j): bit b of word w is lag 32w + b + 1
    auto load_x = [&](uint32_t j, lv (&x)[NW]) {
        const uint32_t o = P - j;
        const uint32_t* r = ((qs[j >> 5] >> (j & 31u)) & 1u ? R1 : R0) + (o >> 5);
#pragma unroll
        for (int n = 0; n < NW; ++n) x[n] = lv_funnel(lv_load(r + 32 * n), lv_load(r + 32 * n + 1), o & 31u);
    };
    auto any = [&](const lv (&e)[NW]) {
        lv a = e[0];
#pragma unroll
        for (int n = 1; n < NW; ++n) a = a | e[n];
        return lv_ballot(a) != 0u;
    };
    auto store_set = [&](uint32_t i, const lv (&e)[NW]) {
        uint32_t* p = ring + (i & (D - 1u)) * (32u * NW);
#pragma unroll
        for (int n = 0; n < NW; ++n) lv_store(p + 32 * n, e[n]);
    };
    auto keep_set = [&](uint32_t i, const lv (&e)[NW]) {
        store_set(i, e);
        if ((i & (gap - 1u)) == 0u) {
            uint32_t* p = kept + i / gap * (32u * NW);
#pragma unroll
            for (int n = 0; n < NW; ++n) lv_store(p + 32 * n, e[n]);
        }
    };
    auto smallest_lag = [&](const lv (&e)[NW]) {   // e is not empty
        uint32_t b = lv_ballot(e[0]), n0 = 0;
        lv x = e[0];
#pragma unroll
        for (int n = 1; n < NW; ++n)
            if (!b) { b = lv_ballot(e[n]); x = e[n]; n0 = (uint32_t)n; }
        const uint32_t lane = ctz32(b);
        return 32u * (lane + 32u * n0) + ctz32(lv_from(x, lane)) + 1u;
    };

    // Whether lag d agrees with the whole of the keys up to t - d, a word per lane.
    auto reaches_start = [&](uint32_t t, uint32_t d) {
        const uint32_t p = t - d, last = p >> 5;
        bool same = true;
        for (uint32_t w0 = 0; w0 <= last && same; w0 += 32u) {
            lv differs = lv_all(0u);
            RM_LANES(l) {
                const uint32_t w = w0 + l, q = (d >> 5) + w;
                if (w <= last) {
                    const uint32_t x = ks[w] ^ funnel32(qs[q], qs[q + 1u], d & 31u);
                    lv_at(differs, l) = w < last ? x : x & (0xFFFFFFFFu >> (31u - (p & 31u)));
                }
            }
            same = lv_ballot(differs) == 0u;
        }
        return same;
    };

    lv E[NW], back[NW], wa[NW], wb[NW];   // wa / wb: the words of R1 that the funnel of the current 32 steps reads
    {
        const uint32_t* r = R1 + ((P - t0) >> 5);
#pragma unroll
        for (int n = 0; n < NW; ++n) {
            E[n] = lv_all(0u); back[n] = lv_all(0u);
            wa[n] = lv_load(r + 32 * n); wb[n] = lv_load(r + 32 * n + 1);
        }
    }
    uint32_t q_word = qs[t0 >> 5];
    // E and back over step t; lags above t are not masked out here (E is a subset of a masked set)
    auto advance = [&](uint32_t t) {
        const uint32_t o = P - t, sh = o & 31u;
        if (sh == 31u) {
            const uint32_t* r = R1 + (o >> 5);
#pragma unroll
            for (int n = 0; n < NW; ++n) { wb[n] = wa[n]; wa[n] = lv_load(r + 32 * n); }
        }
        if (sh == 0u) q_word = qs[t >> 5];
        const uint32_t m = ((q_word >> (t & 31u)) & 1u) - 1u;
#pragma unroll
        for (int n = 0; n < NW; ++n) {
            const lv x = lv_xor(lv_funnel(wa[n], wb[n], sh), m);
            E[n] = E[n] & x;
            back[n] = back[n] & x;
        }
    };

    // the window is [s, t]: front S(s..mid) when s <= mid (ring: sets s..hi), back the steps after mid
    uint32_t s = t0, mid = t0, hi = t0;
    bool have_front = false;
    uint32_t t = t0;
    lv lag;                              // d(t) of the current 32 steps, a step per lane
    auto set_lag = [&](uint32_t first, uint32_t n, uint32_t d) {
        RM_LANES(l) if (l - (first & 31u) < n) lv_at(lag, l) = d;
    };
    while (t < t1) {
        const uint32_t word_end = t1 - t < 32u ? t1 : t + 32u;   // t is a multiple of 32 here
        lag = lv_all(0u);
        while (t < word_end) {
            advance(t);
            bool found = any(E);
            if (!found && have_front) {
                lv F[NW];
                while (!found && s < mid) {
                    ++s;
                    if (s > hi) {   // the ring holds no more of the window: again from the next kept set (or from mid) down to s
                        lv x[NW];
                        uint32_t j = (s & ~(gap - 1u)) + gap;
                        const bool from_kept = j <= mid;
                        const uint32_t* p = kept + j / gap * (32u * NW);
#pragma unroll
                        for (int n = 0; n < NW; ++n) F[n] = from_kept ? lv_load(p + 32 * n) : lv_all(0xFFFFFFFFu);
                        const uint32_t top = from_kept ? j - 1u : mid;
                        for (j = top; ; --j) {
                            load_x(j, x);
#pragma unroll
                            for (int n = 0; n < NW; ++n) F[n] = F[n] & x[n];
                            if (j - s < D) store_set(j, F);
                            if (j == s) break;
                        }
                        hi = top - s < D ? top : s + D - 1u;
                    } else {
                        const uint32_t* p = ring + (s & (D - 1u)) * (32u * NW);
#pragma unroll
                        for (int n = 0; n < NW; ++n) F[n] = lv_load(p + 32 * n);
                    }
#pragma unroll
                    for (int n = 0; n < NW; ++n) E[n] = F[n] & back[n];
                    found = any(E);
                }
                if (!found) {
                    have_front = false;
                    if (mid + 1u < t) {   // the window (mid, t]; for mid + 1 = t the rebuild below starts with that set
                        lv x[NW];
                        load_x(mid + 1u, x);
#pragma unroll
                        for (int n = 0; n < NW; ++n) E[n] = back[n] & x[n];
                        found = any(E);
                    }
                }
            }
            if (!found) {
                lv S[NW], x[NW];
                load_x(t, S);
                found = any(S);
                uint32_t i = t + 1u;        // S = the set of step i, stored, once found
                if (found) keep_set(--i, S);
                bool whole = false;
                uint32_t look = t == t0 ? 32u : ~0u;   // length of the window from which on S is tested as follows
                for (bool more = found; more;) {   // four steps at a time; X(0) is empty: the loop ends there at the latest
                    if (t + 1u - i >= look) {
                        look *= 2u;
                        // No lag agrees over as many steps as the smallest one of S if that agrees to the very first key: the
                        // others of S have fewer keys left, the rest ended before step i.  It is the whole set of the window
                        // then, and there is no front to build: a stream that repeats itself without a flip would go down to
                        // its first step here in every piece (512 streams of 2048 steps 0.63 ms, now 0.07).  Only at the first
                        // step of a piece: where such a lag ends there is no front to go on with, and with a flip in a thousand
                        // steps that happened once per period (1024 streams of 8192 steps 3.8 ms, so 30).
                        const uint32_t d = smallest_lag(S);
                        if (reaches_start(t, d)) {
                            whole = true;
#pragma unroll
                            for (int n = 0; n < NW; ++n)
                                RM_LANES(l) lv_at(S[n], l) = 32u * (uint32_t)n + l == (d - 1u) >> 5 ? 1u << ((d - 1u) & 31u) : 0u;
                            break;
                        }
                    }
                    lv A[4][NW];
#pragma unroll
                    for (uint32_t j = 0; j < 4u; ++j) {
                        load_x(i > j ? i - j - 1u : 0u, x);
#pragma unroll
                        for (int n = 0; n < NW; ++n) A[j][n] = (j ? A[j ? j - 1u : 0u][n] : S[n]) & x[n];
                    }
                    more = any(A[3]);
#pragma unroll
                    for (uint32_t j = 0; j < 4u; ++j) {
                        if (!more && (j == 3u || !any(A[j]))) break;
                        keep_set(--i, A[j]);
#pragma unroll
                        for (int n = 0; n < NW; ++n) S[n] = A[j][n];
                    }
                }
#pragma unroll
                for (int n = 0; n < NW; ++n) E[n] = S[n];
                s = i;                      // t + 1 when X(t) is empty
                mid = t;
                have_front = found && !whole;
                hi = mid - s < D ? mid : s + D - 1u;
#pragma unroll
                for (int n = 0; n < NW; ++n) back[n] = lv_all(0xFFFFFFFFu);
            }
            if (!found) {                   // no key equals q_t so far
                ++t;
                continue;
            }
            // The smallest lag stays the answer for as long as it matches: how long that is comes from 32 bits of q and k,
            // and until then the sets only have to follow.
            const uint32_t d = smallest_lag(E), p = t - d;
            const uint32_t diff = funnel32(qs[t >> 5], qs[(t >> 5) + 1u], t & 31u) ^ funnel32(ks[p >> 5], ks[(p >> 5) + 1u], p & 31u);
            uint32_t same = diff ? ctz32(diff) : 32u;
            if (same > word_end - t) same = word_end - t;
            set_lag(t, same, d);
            const uint32_t end = t + same;
            for (++t; t < end; ++t) advance(t);
        }
        lv bit;
        const uint32_t w = (t - 1u) >> 5;
        RM_LANES(l) {
            const uint32_t d = lv_at(lag, l), r = 32u * w + l - d + 1u;
            lv_at(bit, l) = d ? (vw[r >> 5] >> (r & 31u)) & 1u : 0u;
        }
        const uint32_t out = lv_ballot(bit);
        RM_LANES(l) if (l == 0u) idx[w] = out;
    }
}

}  // namespace match
}  // namespace ullis
