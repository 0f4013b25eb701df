// 1-bit ROSA match by contexts: the idx of RosaSam::push (src/rosa.rs:100-176), every step by itself.
//
// What a step needs (rosa_match.cuh says why) is the position r < t whose key history agrees with the query history
// of step t over the most steps, the latest one of equals.  The keys are put into buckets by a property of their
// latest bits (a stable counting sort, so a bucket lists its positions in ascending order), and a step compares its
// history, 32 steps at a time, with those of the positions of its bucket that lie before t.  Two properties:
//
//  * the last `c` bits, about 8 positions per bucket where both bits are common.  Only where the bucket holds no
//    position before t is the longest agreement shorter than c; the neighbouring buckets that share ever fewer of the
//    latest bits are looked through then.
//  * the length of the run of equal bits that ends at the position, where one bit is rare: every run has one position
//    per length, so a bucket holds no more positions than there are runs.  Without a position of equal run length
//    before t the agreement ends inside a run; then the latest position with a run at least as long counts, or else
//    the longest run, and both are found through the longest runs of the words (`Runs`).
//
// The product of key and query counts over the buckets says how much either costs before any comparison is made; a
// stream that is too expensive both ways is left to rosa_match.cuh.
#pragma once
#include <stdint.h>

#if defined(__CUDACC__)
#define RC_HD __device__ __forceinline__
#else
#define RC_HD inline
#endif

namespace ullis {
namespace context {

// Context length: about 8 positions per bucket on evenly spread keys.
#if defined(__CUDACC__)
__host__ __device__
#endif
inline uint32_t bits_for(uint32_t T) {
    uint32_t c = 0;
    while (T >> (c + 4u)) ++c;      // floor(log2 T) - 3
    return c < 2u ? 2u : c > 12u ? 12u : c;
}

// The same for a stream whose steps find many positions in their buckets: one bit more, so that the large ones halve.  Above 4096
// steps (6000, biased streams) the sort takes what that saves.
#if defined(__CUDACC__)
__host__ __device__
#endif
inline uint32_t bits_for_uneven(uint32_t T) { return bits_for(T) + (T <= 4096u ? 1u : 0u); }

constexpr uint32_t BRUTE = 64;      // steps below this compare with every earlier position

struct alignas(8) Entry {           // a position and the 32 key bits that end there
    uint32_t key, r;
};

// The 32 bits that end with bit i of a stream, bit i on top; W[0] = 0 and W[1 + j] = word j, so bits before the first
// one read as zeros.
RC_HD uint32_t window(const uint32_t* W, uint32_t i) {
    const uint32_t lo = W[i >> 5], hi = W[(i >> 5) + 1u], sh = 31u - (i & 31u);
#if defined(__CUDACC__)
    return __funnelshift_l(lo, hi, sh);
#else
    return sh ? hi << sh | lo >> (32u - sh) : hi;
#endif
}
RC_HD uint32_t leading(uint32_t x) {   // leading zeros, 32 for 0
#if defined(__CUDACC__)
    return (uint32_t)__clz((int)x);
#else
    return x ? (uint32_t)__builtin_clz(x) : 32u;
#endif
}

// Number of steps over which the histories of q at t and of k at r agree (r < t), x = the xor of their windows.
RC_HD uint32_t agreement(const uint32_t* Q, const uint32_t* K, uint32_t t, uint32_t r, uint32_t x, uint32_t& deep) {
    uint32_t n = leading(x);
    if (n == 32u) {
        while (n <= r) {
            const uint32_t l = leading(window(Q, t - n) ^ window(K, r - n));
            n += l;
            ++deep;
            if (l < 32u) break;
        }
    }
    return n < r + 1u ? n : r + 1u;
}

// Length of the run of equal bits that ends with bit i; ends[w] = the one that ends with the last bit of word w - 1.
RC_HD uint32_t run_at(const uint32_t* W, const uint16_t* ends, uint32_t i) {
    const uint32_t x = window(W, i), in_word = (i & 31u) + 1u;
    const uint32_t n = leading((x >> 31) ? ~x : x);
    if (n < in_word || i < 32u) return n < in_word ? n : in_word;
    const bool same = ((W[i >> 5] ^ x) >> 31) == 0u;           // W[i >> 5] is the word before
    return in_word + (same ? ends[i >> 5] : 0u);
}
// ends[w] for w >= 1
RC_HD uint32_t run_at_end(const uint32_t* W, uint32_t w) {
    const uint32_t fill = (W[w] >> 31) ? 0xFFFFFFFFu : 0u;
    uint32_t n = 0;
    while (w >= 1u && W[w] == fill) { n += 32u; --w; }
    return w >= 1u ? n + leading(W[w] ^ fill) : n;
}
RC_HD uint32_t bit_at(const uint32_t* W, uint32_t i) { return (W[(i >> 5) + 1u] >> (i & 31u)) & 1u; }
RC_HD uint32_t run_key(const uint32_t* W, const uint16_t* ends, uint32_t i, uint32_t c) {
    const uint32_t half = 1u << (c - 1u);
    return bit_at(W, i) * half + (run_at(W, ends, i) & (half - 1u));
}

// What the runs of a stream are looked up by.  in_word[b * words + w]: the longest run of bit b that ends at a position
// of word w; before[b * words + w]: the longest one that ends in an earlier word, as length << 16 | position + 1 with
// the latest position of equals (0: none).
struct Runs {
    const uint16_t *ends, *in_word;
    const uint32_t* before;
};
// The longest run of bit b that ends in word w (positions below T), in the form of `before`.
RC_HD uint32_t longest_in_word(const uint32_t* W, const uint16_t* ends, uint32_t w, uint32_t T, uint32_t b) {
    uint32_t best = 0;
    for (uint32_t i = T < 32u * w + 32u ? T : 32u * w + 32u; i > 32u * w;) {
        const uint32_t n = run_at(W, ends, i - 1u);
        if (bit_at(W, i - 1u) == b && n > best >> 16) best = n << 16 | i;
        if (n >= i) break;
        i -= n;
    }
    return best;
}

// Of the positions among entries [b, e), every step-th, that lie before t and have the query's run length: the longest
// agreement beyond the run, packed as agreement << 16 | position + 1 with the latest of equals (0: none).
RC_HD uint32_t scan_runs(const Entry* entries, uint32_t b, uint32_t e, uint32_t step, const uint32_t* Q, const uint32_t* K, const Runs& R, uint32_t run,
                         uint32_t t, uint32_t& deep) {
    uint32_t best = 0;
    if (run > t) return 0u;                                    // beyond the run there is no more of the query history
    const uint32_t wq = window(Q, t - run);
    for (; b < e; b += step) {
        const uint32_t r = entries[b].r;
        if (r >= t) break;
        if (r < run || run_at(K, R.ends, r) != run) continue;
        const uint32_t v = agreement(Q, K, t - run, r - run, wq ^ window(K, r - run), deep) << 16 | (r + 1u);   // at least 1
        best = v > best ? v : best;
    }
    return best;
}
// Without such a position: the latest one before t whose run of this bit reaches `run`, else the latest of the longest
// runs, as r + 1.
RC_HD uint32_t find_inside_run(const uint32_t* K, const Runs& R, uint32_t words, uint32_t bit, uint32_t run, uint32_t t, uint32_t& deep) {
    uint32_t best = 0, at = 0, w = t >> 5;
    for (uint32_t i = t; i > 32u * w;) {                       // the positions in the word of t
        const uint32_t n = run_at(K, R.ends, i - 1u);
        if (bit_at(K, i - 1u) == bit) {
            if (n >= run) return i;
            if (n > best) { best = n; at = i; }
        }
        if (n >= i) break;
        i -= n;
    }
    const uint32_t longest = R.before[bit * words + w];
    if (longest >> 16 <= run) return longest >> 16 > best ? longest & 0xFFFFu : at;
    do { --w; ++deep; } while (R.in_word[bit * words + w] < run);   // there is one
    for (uint32_t i = 32u * w + 32u;;) {
        const uint32_t n = run_at(K, R.ends, i - 1u);
        if (bit_at(K, i - 1u) == bit && n >= run) return i;
        i -= n;
    }
}

// The positions before t of the buckets [first, first + n): the smallest of top << 16 - position, top = the highest bit
// in which the windows differ (-1: none) and at least 30 - position (a history has position + 1 steps).
RC_HD int32_t scan(const Entry* entries, const uint16_t* start, uint32_t first, uint32_t n, uint32_t t, uint32_t wq, int32_t best) {
    uint32_t b = start[first];
    for (uint32_t x = first + 1u; x <= first + n; ++x) {
        const uint32_t e = start[x];
        const Entry* p = entries + b;
        const Entry* const end = entries + e;
        while (p < end && p->r < 31u && p->r < t) {
            const int32_t top = 31 - (int32_t)leading(wq ^ p->key), least = 30 - (int32_t)p->r;
            const int32_t v = (top > least ? top : least) * 65536 - (int32_t)p->r;
            best = v < best ? v : best;
            ++p;
        }
        while (p < end) {
            const Entry a = *p++;
            if (a.r >= t) break;
            const int32_t v = (31 - (int32_t)leading(wq ^ a.key)) * 65536 - (int32_t)a.r;
            best = v < best ? v : best;
        }
        b = e;
    }
    return best;
}
// One position of them.
RC_HD int32_t scan_one(Entry a, uint32_t t, uint32_t wq, int32_t best) {
    if (a.r >= t) return best;
    const int32_t top = 31 - (int32_t)leading(wq ^ a.key), least = 30 - (int32_t)a.r;
    const int32_t v = (top > least ? top : least) * 65536 - (int32_t)a.r;
    return v < best ? v : best;
}
// The same where the positions of a bucket are known to agree in equally many bits: the latest one of each counts, found
// by bisection (a bucket beside the query's own can be as large as the stream).  From bucket to bucket by the keys, past the
// empty ones: where a bit is rare nearly all of them are (64 sequences of the default model, contexts 8.7 -> 7.5 ms in all).
RC_HD int32_t scan_latest(const Entry* entries, const uint16_t* start, uint32_t c, uint32_t first, uint32_t n, uint32_t t, uint32_t wq,
                          int32_t best) {
    const uint32_t end = start[first + n];
    for (uint32_t b = start[first]; b < end;) {
        const uint32_t e = start[(entries[b].key >> (32u - c)) + 1u];
        uint32_t lo = b, hi = e;                               // entries below lo lie before t, from hi on they do not
        while (lo < hi) {
            const uint32_t m = (lo + hi) >> 1;
            if (entries[m].r < t) lo = m + 1u; else hi = m;
        }
        if (lo > b) {
            const Entry a = entries[lo - 1u];
            const int32_t top = 31 - (int32_t)leading(wq ^ a.key), least = 30 - (int32_t)a.r;
            const int32_t v = (top > least ? top : least) * 65536 - (int32_t)a.r;
            best = v < best ? v : best;
        }
        b = e;
    }
    return best;
}
RC_HD uint32_t scan_position(int32_t best) { return (uint32_t)-best & 0xFFFFu; }
RC_HD int32_t scan_agreement(int32_t best) { return 31 - ((best + (int32_t)scan_position(best)) >> 16); }   // -1: no position

constexpr int32_t SCAN_NOTHING = 32 * 65536;
RC_HD bool scan_full(int32_t best) { return best <= -65536; }   // a whole window agrees

// Where the search for step t begins: with `wide` sets of as many context bits as leave 2 to 4 positions before t on
// evenly spread keys (4 to 8: contexts of 16 sequences in training 6.07 ms, not 5.80), otherwise with all c bits - the
// buckets [first, first + n).
struct Query {
    uint32_t wq, ctx, l, first, n;
};
RC_HD Query query(const uint32_t* Q, uint32_t c, bool wide, uint32_t t) {
    Query z;
    z.wq = window(Q, t);
    z.ctx = z.wq >> (32u - c);
    z.l = c;
    if (wide && 30u - leading(t) < c) z.l = 30u - leading(t);  // floor(log2 t) - 1
    z.first = z.ctx >> (c - z.l) << (c - z.l);
    z.n = 1u << (c - z.l);
    return z;
}

// Agreements counted on beyond the windows: of the positions before t among entries [b, e), every step-th, whose window is
// wq; packed as in scan_runs.  Ends when `deep` passes `most`: the stream is given up then, whatever the answer.
RC_HD uint32_t scan_deep(const Entry* entries, uint32_t b, uint32_t e, uint32_t step, const uint32_t* Q, const uint32_t* K, uint32_t wq, uint32_t t,
                         uint32_t& deep, uint32_t most) {
    uint32_t best = 0;
    for (; b < e && deep <= most; b += step) {
        const Entry a = entries[b];
        if (a.r >= t || wq != a.key) continue;
        const uint32_t v = agreement(Q, K, t, a.r, 0u, deep) << 16 | (a.r + 1u);
        best = v > best ? v : best;
    }
    return best;
}

// r + 1 for a step below BRUTE, 0 without a match.
RC_HD uint32_t find_brute(const uint32_t* Q, const uint32_t* K, uint32_t t, uint32_t& deep) {
    const uint32_t wq = window(Q, t);
    uint32_t best = 0;
    for (uint32_t r = 0; r < t; ++r) {
        const uint32_t n = agreement(Q, K, t, r, wq ^ window(K, r), deep), v = n << 16 | (r + 1u);
        best = n && v > best ? v : best;
    }
    return best & 0xFFFFu;
}

// r + 1 for step t >= BRUTE, 0 without a match; best: what scan() found in the query's own buckets, not scan_full().
// Whatever has not been looked at when the search ends agrees in fewer bits than the best.  (A position with a history
// shorter than a context lies in the bucket of that history filled up with zeros, which agrees with the query in no fewer
// bits than the history itself.)
RC_HD uint32_t find_shorter(const Entry* entries, const uint16_t* start, uint32_t c, const Query& z, uint32_t t, int32_t best) {
    uint32_t l = z.l;
    while (scan_agreement(best) < (int32_t)l && --l > 0u) {    // the buckets that agree in l bits and differ in the next
        const uint32_t sh = c - 1u - l;
        best = scan_latest(entries, start, c, ((z.ctx >> sh) ^ 1u) << sh, 1u << sh, t, z.wq, best);
    }
    return scan_agreement(best) > 0 ? scan_position(best) + 1u : 0u;
}

}  // namespace context
}  // namespace ullis
