// RosaSam::push (src/rosa.rs:100-176) for streams that advance one step per call, without an automaton.
//
// rosa_match.cuh says what a push computes: the position r < i whose key history agrees with the query history of
// step i over the most steps, the latest of equals, and the v bit after it.  While the lag of the step before still
// matches it stays the answer (the matches of step i are those of step i - 1 that go on), which is one bit to look at;
// otherwise the positions of a key word that agree with the query history are a bit mask, refined by one step of the
// histories after the other - a word per lane where a warp searches for one stream, word after word where each lane has
// a stream of its own - and only where 32 steps agree are they counted on one by one.  A stream is its three bit
// histories and a lag: 3 * T / 8 + 16 bytes (at T = 2048 784 instead of the 28.7 KB of an automaton with its
// chain), and the cost of a step grows with i / 32 and not with the runs of the keys.
#pragma once
#include <stdint.h>

namespace ullis {
namespace push {

// Per stream: the lag of the last step (0: no match), the last 32 query bits (the latest on top), and the words of k
// and v that are being filled.
struct alignas(16) Current {
    uint32_t lag, q, k, v;
};

// The histories of all streams, stream by stream: words of q, then of k, then of v (whole words only).
struct Histories {
    Current* current;
    uint32_t* words;
    size_t wps;
    __device__ const uint32_t* of(size_t stream, int which) const { return words + (stream * 3 + which) * wps; }
};

// 32 bits that end with bit p of a history whose word `last` is still in a register.
__device__ __forceinline__ uint32_t window(const uint32_t* words, uint32_t last, uint32_t current, uint32_t p) {
    const uint32_t w = p >> 5;
    const uint32_t hi = w == last ? current : words[w], lo = w ? words[w - 1u] : 0u;
    return __funnelshift_l(lo, hi, 31u - (p & 31u));
}

// Steps on which the histories that end at step i of the queries and at position r of the keys agree, from n on.
__device__ __forceinline__ uint32_t agreement(const uint32_t* q, const uint32_t* k, uint32_t last, uint32_t q_word,
                                              uint32_t k_word, uint32_t i, uint32_t r, uint32_t n) {
#pragma unroll 1
    while (n <= r) {
        const uint32_t same = (uint32_t)__clz((int)(window(q, last, q_word, i - n) ^ window(k, last, k_word, r - n)));
        n += same;
        if (same < 32u) break;
    }
    return min(n, r + 1u);
}

// The lag of step i by the whole warp where the last 32 query bits are equal (c); 0: fewer than 32 steps agree anywhere.
// Streams that hardly ever change come here at almost every step, with whole windows of equal bits at most positions, so
// these are not compared one by one but as runs: with n the run of c at step i, a position at the end of a shorter run of
// c among the keys agrees on just that run, one with a longer run on n, and only one whose run is n long on more.  A lane
// has a word; a run of 32 or more that ends in it covers its lowest bits, and the words before say how much goes before
// them.  (64 sequences of the default model with nearly constant channels, position 2 000: 69 ms a step position by
// position, by the runs of the keys 1.8 ms.)
__device__ __forceinline__ uint32_t search_runs(const uint32_t* q, const uint32_t* k, uint32_t i, uint32_t wq, uint32_t k_word) {
    const uint32_t lane = threadIdx.x & 31u, last = i >> 5, q_word = wq >> (31u - (i & 31u));
    uint32_t n_run = (i & 31u) + 1u;
#pragma unroll 1
    for (uint32_t w1 = last;; w1 -= 32u) {                       // words of c below w1
        const uint32_t y = lane < w1 ? q[w1 - 1u - lane] ^ ~wq : 0u, full = __ballot_sync(0xFFFFFFFFu, y == ~0u);
        if (full == ~0u) { n_run += 1024u; continue; }
        const uint32_t l = (uint32_t)__ffs((int)~full) - 1u;
        n_run += 32u * l + (uint32_t)__clz((int)~__shfl_sync(0xFFFFFFFFu, y, (int)l));
        break;
    }
    uint32_t longest = 0, position = 0, before = 0;              // before: run of c that ends at the last word so far
#pragma unroll 1
    for (uint32_t w0 = 0; w0 <= last; w0 += 32u) {
        const uint32_t w = w0 + lane;
        const uint32_t x = w < last ? k[w] ^ ~wq : w == last ? (k_word ^ ~wq) & ((1u << (i & 31u)) - 1u) : 0u;
        const uint32_t full = __ballot_sync(0xFFFFFFFFu, x == ~0u), upper = (uint32_t)__clz((int)~x);
        const uint32_t lower = x == ~0u ? 32u : (uint32_t)__ffs((int)~x) - 1u;
        const uint32_t z = lane ? min((uint32_t)__clz((int)(~full << (32u - lane))), lane) : 0u;   // words of c right below
        const uint32_t there = __shfl_sync(0xFFFFFFFFu, upper, (int)(z < lane ? lane - 1u - z : 0u));
        const uint32_t carry = 32u * z + (z < lane ? there : before), run = carry + lower;
        if (run >= 32u && lower) {
            if (carry < n_run && n_run <= run) {
                const uint32_t r = 32u * w + n_run - carry - 1u, n = agreement(q, k, last, q_word, k_word, i, r, n_run);
                if (n >= longest) { longest = n; position = r; }
            }
            if (run != n_run && min(run, n_run) >= longest) { longest = min(run, n_run); position = 32u * w + lower - 1u; }
        }
        const uint32_t h = 31u - (uint32_t)__clz((int)~full);   // full == ~0: h = -1
        const uint32_t top = __shfl_sync(0xFFFFFFFFu, upper, (int)(full == ~0u ? 0u : h));
        before = full == ~0u ? before + 1024u : 32u * (31u - h) + top;
    }
    const uint32_t top = __reduce_max_sync(0xFFFFFFFFu, longest);
    if (top < 32u) return 0u;
    return i - __reduce_max_sync(0xFFFFFFFFu, longest == top ? position : 0u);
}

// Of the positions `valid` of a word of keys those whose histories agree with the query history wq over the most steps, up to 32; `before`:
// the word before.  MAYBE_FIRST: position r of the first word (others = 0; ~0 in any other) has only r + 1 steps behind it.
// (A position at a time - window, difference, leading zeros - took four instructions for each of 32 positions; a word takes 32 for
// the first eight steps, and few words have positions beyond.)
struct Agreeing {
    uint32_t steps, positions;
};
template <bool MAYBE_FIRST>
__device__ __forceinline__ Agreeing agreeing(uint32_t before, uint32_t word, uint32_t valid, uint32_t wq, uint32_t others) {
    Agreeing z{0u, 0u};
    uint32_t at = valid;
#pragma unroll
    for (uint32_t d = 1; d <= 8u; ++d) {
        at &= ~(__funnelshift_l(before, word, d - 1u) ^ (uint32_t)((int32_t)(wq << (d - 1u)) >> 31));
        const uint32_t full = MAYBE_FIRST ? at & (0xFFFFFFFFu << (d - 1u) | others) : at;
        if (full) z = Agreeing{d, full};
    }
#pragma unroll 1
    for (uint32_t d = 9; at && d <= 32u; ++d) {
        at &= ~(__funnelshift_l(before, word, d - 1u) ^ (uint32_t)((int32_t)(wq << (d - 1u)) >> 31));
        const uint32_t full = MAYBE_FIRST ? at & (0xFFFFFFFFu << (d - 1u) | others) : at;
        if (full) z = Agreeing{d, full};
    }
    return z;
}
__device__ __forceinline__ uint32_t top_bit(uint32_t x) { return 31u - (uint32_t)__clz((int)x); }

// The lag of step i for one stream, by the whole warp; wq: the query bits up to i, k_word: the keys before i.
__device__ __forceinline__ uint32_t search(const uint32_t* q, const uint32_t* k, uint32_t i, uint32_t wq, uint32_t k_word) {
    const uint32_t lane = threadIdx.x & 31u, last = i >> 5, q_word = wq >> (31u - (i & 31u));
    if (i >= 32u && (wq == 0u || wq == ~0u)) {
        const uint32_t lag = search_runs(q, k, i, wq, k_word);
        if (lag) return lag;
    }
    uint32_t best = 0, bit = 0, carry = 0;      // agreement << 26 | word of the position; the bit within the word
#pragma unroll 1
    for (uint32_t w0 = 0; w0 <= last; w0 += 32u) {
        const uint32_t w = w0 + lane, mine = w < last ? k[w] : w == last ? k_word : 0u;
        const uint32_t below = __shfl_up_sync(0xFFFFFFFFu, mine, 1);
        const uint32_t valid = w < last ? ~0u : w == last ? (1u << (i & 31u)) - 1u : 0u;   // not a key yet
        const Agreeing z = agreeing<true>(lane ? below : carry, mine, valid, wq, w ? ~0u : 0u);
        if (z.steps && (z.steps << 26 | w) >= best) {
            best = z.steps << 26 | w;
            bit = top_bit(z.positions);
        }
        carry = __shfl_sync(0xFFFFFFFFu, mine, 31);
    }
    const uint32_t most = __reduce_max_sync(0xFFFFFFFFu, best);
    if (most >> 26 < 32u) {
        const uint32_t w = most & 0x3FFFFFFu;
        bit = __shfl_sync(0xFFFFFFFFu, bit, (int)(w & 31u));   // of the lane that has this word
        return most ? i - (32u * w + bit) : 0u;
    }
    // whole windows agree: count on from there
    uint32_t longest = 0, position = 0;
#pragma unroll 1
    for (uint32_t r = lane; r < i; r += 32u) {
        if (window(k, last, k_word, r) != wq) continue;
        const uint32_t n = agreement(q, k, last, q_word, k_word, i, r, 32u);
        if (n >= longest) { longest = n; position = r; }
    }
    const uint32_t top = __reduce_max_sync(0xFFFFFFFFu, longest);
    return i - __reduce_max_sync(0xFFFFFFFFu, longest == top ? position : 0u);
}

// The same for one stream per lane (open lanes only); DEEP where whole windows agree, which is left to search().
constexpr uint32_t DEEP = ~0u;
__device__ __forceinline__ uint32_t search_alone(const uint32_t* k, uint32_t i, uint32_t wq, uint32_t k_word) {
    const uint32_t last = i >> 5;
    uint32_t steps = 0, position = 0, word = k_word, valid = (1u << (i & 31u)) - 1u;
#pragma unroll 1
    for (uint32_t w = last; steps < 32u; --w) {   // from the latest word on: of equals the first one found counts
        const uint32_t before = w ? k[w - 1u] : 0u;
        const Agreeing z = w ? agreeing<false>(before, word, valid, wq, ~0u) : agreeing<true>(before, word, valid, wq, 0u);
        if (z.steps > steps) {
            steps = z.steps;
            position = 32u * w + top_bit(z.positions);
        }
        if (w == 0u) break;
        word = before;
        valid = ~0u;
    }
    return steps == 32u ? DEEP : steps ? i - position : 0u;
}

// What step i of 32 streams (first + lane; a lane with live = false has none) can know before its bits: whether the lag of
// the step before goes on if q is 1, and the v bit that it leads to (of the word being filled for lag 1: not known yet).
struct Ahead {
    Current c;
    uint32_t key, value;
};
__device__ __forceinline__ Ahead begin(const Histories& H, size_t first, bool live, uint32_t i) {
    Ahead a{{0u, 0u, 0u, 0u}, 0u, 0u};
    const size_t s = first + (threadIdx.x & 31u);
    if (!live || i == 0u) return a;
    a.c = H.current[s];
    if ((i & 31u) == 0u) a.c.k = a.c.v = 0u;
    if (a.c.lag) {
        const uint32_t p = i - a.c.lag, last = i >> 5;
        a.key = ((p >> 5 == last ? a.c.k : H.of(s, 1)[p >> 5]) >> (p & 31u)) & 1u;
        a.value = ((p + 1u) >> 5 == last ? a.c.v : H.of(s, 2)[(p + 1u) >> 5]) >> ((p + 1u) & 31u) & 1u;
    }
    return a;
}

// Step i of the same streams: returns idx of the lane's stream.
__device__ __forceinline__ bool step(const Histories& H, size_t first, bool live, uint32_t i, Ahead a, uint32_t qb, uint32_t kb, uint32_t vb) {
    const uint32_t lane = threadIdx.x & 31u, b = i & 31u, last = i >> 5;
    const size_t s = first + lane;
    Current c = a.c;
    c.q = c.q >> 1 | qb << 31;
    c.v |= vb << b;
    const bool goes_on = c.lag && a.key == qb;
    const bool known = !live || goes_on;
    uint32_t open = __ballot_sync(0xFFFFFFFFu, !known);
    // One after the other by the whole warp, or side by side with a lane each: by the instructions either takes.
    if ((uint32_t)__popc(open) * (60u * (last / 32u + 1u) + 110u) > 48u * (last + 1u) + 60u) {
        if (!known) c.lag = search_alone(H.of(s, 1), i, c.q, c.k);
        open = __ballot_sync(0xFFFFFFFFu, !known && c.lag == DEEP);
    }
    while (open) {
        const int l = __ffs((int)open) - 1;
        open &= open - 1u;
        const uint32_t lag = search(H.of(first + l, 0), H.of(first + l, 1), i, __shfl_sync(0xFFFFFFFFu, c.q, l),
                                    __shfl_sync(0xFFFFFFFFu, c.k, l));
        if ((int)lane == l) c.lag = lag;
    }
    bool bit = false;
    if (live) {
        if (goes_on && c.lag > 1u) {
            bit = a.value != 0u;
        } else if (c.lag) {
            const uint32_t p = i - c.lag + 1u;
            const uint32_t word = p >> 5 == last ? c.v : H.of(s, 2)[p >> 5];
            bit = ((word >> (p & 31u)) & 1u) != 0u;
        }
        c.k |= kb << b;
        H.current[s] = c;
        if (b == 31u) {
            uint32_t* words = H.words + s * 3 * H.wps + last;
            words[0] = c.q;
            words[H.wps] = c.k;
            words[2 * H.wps] = c.v;
        }
    }
    return bit;
}

}  // namespace push
}  // namespace ullis
