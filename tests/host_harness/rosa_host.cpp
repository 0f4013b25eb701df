// Host-compiled harness around the automaton-free ROSA match (rosa_match.cuh, rosa_context.cuh), used only by the CPU
// tests.  It does with loops what the kernels of sam.cu do around these routines: the stable sort of the keys into
// buckets, the tables of the runs, the pieces of a stream.  It is not part of the shipped library.
#include <cstddef>
#include <cstdint>
#include <cstring>
#include <vector>

#include "../../ullis_b200/csrc/rosa_context.cuh"
#include "../../ullis_b200/csrc/rosa_heads.cuh"
#include "../../ullis_b200/csrc/rosa_match.cuh"

using namespace ullis;

namespace {

constexpr uint32_t POISON = 0xA5A5A5A5u;

// One stream in pieces of `piece` steps, from the last piece to the first.  false: something wrote past its memory.
bool by_lags(const uint32_t* q, const uint32_t* k, const uint32_t* v, uint32_t T, uint32_t piece, uint32_t* out) {
    const uint32_t nw_max = T <= 1024u ? 1u : T <= 2048u ? 2u : T <= 4096u ? 4u : 8u;
    const uint32_t ring_words = nw_max <= 2u ? 1024u : nw_max == 4u ? 2048u : 4096u;
    const match::Layout L(nw_max, ring_words);
    const size_t kept_words = (size_t)match::CHECKPOINTS * 32u * nw_max;
    std::vector<uint32_t> mem(L.total + 32u, POISON), kept(kept_words + 32u, POISON);
    const uint32_t gap = match::checkpoint_gap(T);
    for (uint32_t n = (T + piece - 1u) / piece; n-- > 0u;) {
        const uint32_t t0 = n * piece, t1 = t0 + piece < T ? t0 + piece : T;
        if (t1 > 4096u) match::piece<8>(mem.data(), L, ring_words, kept.data(), gap, q, k, v, out, t0, t1);
        else if (t1 > 2048u) match::piece<4>(mem.data(), L, ring_words, kept.data(), gap, q, k, v, out, t0, t1);
        else if (t1 > 1024u) match::piece<2>(mem.data(), L, ring_words, kept.data(), gap, q, k, v, out, t0, t1);
        else match::piece<1>(mem.data(), L, ring_words, kept.data(), gap, q, k, v, out, t0, t1);
    }
    for (uint32_t i = 0; i < 32u; ++i)
        if (mem[L.total + i] != POISON || kept[kept_words + i] != POISON) return false;
    return true;
}

// One stream by contexts of c bits: by the last bits (wide: few positions before a step, as the easy streams are searched),
// or by the lengths of the runs.
void by_contexts(const uint32_t* q, const uint32_t* k, const uint32_t* v, uint32_t T, uint32_t c, bool by_runs, bool wide, uint32_t* out) {
    using namespace context;
    const uint32_t C = 1u << c, words = (T + 31u) / 32u;
    std::vector<uint32_t> Q(words + 1u, 0u), K(words + 1u, 0u);
    std::memcpy(Q.data() + 1, q, words * 4u);
    std::memcpy(K.data() + 1, k, words * 4u);
    std::vector<uint16_t> q_ends(words + 1u, 0), k_ends(words + 1u, 0), in_word(2u * words), start(C + 2u, 0);
    std::vector<uint32_t> before(2u * words);
    for (uint32_t w = 0; w <= words; ++w) {
        q_ends[w] = (uint16_t)run_at_end(Q.data(), w);
        k_ends[w] = (uint16_t)run_at_end(K.data(), w);
    }
    for (uint32_t b = 0; b < 2u; ++b) {
        uint32_t most = 0;
        for (uint32_t w = 0; w < words; ++w) {
            const uint32_t x = longest_in_word(K.data(), k_ends.data(), w, T, b);
            in_word[b * words + w] = (uint16_t)(x >> 16);
            before[b * words + w] = most;
            if (x > most) most = x;
        }
    }
    const Runs runs{k_ends.data(), in_word.data(), before.data()};
    auto key = [&](const std::vector<uint32_t>& W, const std::vector<uint16_t>& ends, uint32_t i) {
        return by_runs ? run_key(W.data(), ends.data(), i, c) : window(W.data(), i) >> (32u - c);
    };
    std::vector<std::vector<uint32_t>> buckets(C);
    for (uint32_t r = 0; r < T; ++r) buckets[key(K, k_ends, r)].push_back(r);
    std::vector<Entry> entries;
    for (uint32_t x = 0; x < C; ++x) {
        start[x] = (uint16_t)entries.size();
        for (uint32_t r : buckets[x]) entries.push_back(Entry{window(K.data(), r), r});
    }
    start[C] = (uint16_t)T;
    std::memset(out, 0, words * 4u);
    for (uint32_t t = 0; t < T; ++t) {
        uint32_t deep = 0, r1 = 0;
        if (t < BRUTE) {
            r1 = find_brute(Q.data(), K.data(), t, deep);
        } else {
            Query z{};
            uint32_t run = 0;
            if (by_runs) {
                run = run_at(Q.data(), q_ends.data(), t);
                z.wq = window(Q.data(), t);
                z.first = key(Q, q_ends, t);
                z.n = 1u;
            } else {
                z = query(Q.data(), c, wide, t);
            }
            const uint32_t b = start[z.first], e = start[z.first + z.n];
            uint32_t found = 0;
            int32_t best = SCAN_NOTHING;
            if (by_runs && run >= 32u) {
                found = scan_runs(entries.data(), b, e, 1u, Q.data(), K.data(), runs, run, t, deep);
            } else {
                best = scan(entries.data(), start.data(), z.first, z.n, t, z.wq, best);
                if (scan_full(best)) found = scan_deep(entries.data(), b, e, 1u, Q.data(), K.data(), z.wq, t, deep, ~0u);
            }
            if (found) r1 = found & 0xFFFFu;
            else if (!by_runs) r1 = find_shorter(entries.data(), start.data(), c, z, t, best);
            else if (scan_agreement(best) > (int32_t)run) r1 = scan_position(best) + 1u;
            else r1 = find_inside_run(K.data(), runs, words, bit_at(Q.data(), t), run, t, deep);
        }
        if (r1 && ((v[r1 >> 5] >> (r1 & 31u)) & 1u)) out[t >> 5] |= 1u << (t & 31u);
    }
}

// One stream by the latest positions of its contexts, the rows of a warp lane by lane; the keys of the rows before row0 are put
// in without answers.
void by_heads(const uint32_t* q, const uint32_t* k, const uint32_t* v, uint32_t T, uint32_t row0, uint32_t* out) {
    const uint32_t words = (T + 31u) / 32u;
    std::vector<uint32_t> Q(words + 1u, 0u), K(words + 1u, 0u), latest_7(heads::LATEST_7, 0u), latest_3(heads::LATEST_3, 0u);
    std::memcpy(Q.data() + 1, q, words * 4u);
    std::memcpy(K.data() + 1, k, words * 4u);
    std::vector<uint16_t> latest_11(heads::LATEST_11, 0), link(32u * words + 2u, 0);
    for (uint32_t row = 0; row < words; ++row) {
        uint32_t found[32], wk[32], wq[32];
        for (uint32_t l = 0; l < 32u; ++l) {
            wk[l] = context::window(K.data(), 32u * row + l);
            wq[l] = context::window(Q.data(), 32u * row + l);
            found[l] = heads::probe_11(latest_11.data(), wq[l]);
            if (!found[l]) found[l] = heads::probe(latest_7.data(), wq[l], 7u);
            if (!found[l]) found[l] = heads::probe(latest_3.data(), wq[l], 3u);
        }
        for (uint32_t l = 0; l < 32u; ++l) {   // in order, so that the last lane of a context counts
            const uint32_t r1 = 32u * row + l + 1u;
            link[r1] = latest_11[wk[l] >> 21];
            latest_11[wk[l] >> 21] = (uint16_t)r1;
            latest_7[wk[l] >> 25] = latest_3[wk[l] >> 29] = r1;
        }
        if (row < row0) continue;
        out[row] = 0u;
        for (uint32_t l = 0; l < 32u && 32u * row + l < T; ++l) {
            const uint32_t t = 32u * row + l, below = (1u << l) - 1u;
            const uint32_t in_row = row ? heads::agreeing<false>(K[row], K[row + 1u], below, wq[l]) : heads::agreeing<true>(0u, K[1], below, wq[l]);
            if (in_row) {
                const uint32_t near = heads::latest(row, in_row);
                uint32_t bits = context::leading(wq[l] ^ wk[(near - 1u) & 31u]);
                bits = bits < heads::DEPTH ? bits : heads::DEPTH;
                bits = bits < near ? bits : near;
                if (bits >= found[l] >> 16) found[l] = bits << 16 | near;
            }
            uint32_t r1 = found[l] & 0xFFFFu, best = 0, work = 0;
            for (uint32_t p = found[l] >> 16 == heads::DEPTH ? r1 : 0u; p; p = link[p]) {
                uint32_t n = context::leading(wq[l] ^ heads::window_before(K.data(), p));
                if (n > p) n = p;
                if (n == 32u) n = context::agreement(Q.data(), K.data(), t, p - 1u, 0u, work);
                if (n > best) {
                    best = n;
                    r1 = p;
                }
            }
            if (r1 && ((v[r1 >> 5] >> (r1 & 31u)) & 1u)) out[row] |= 1u << l;
        }
    }
}

}  // namespace

// way: 0 = contexts by the last bits, 1 = the same with every bit of a context, 2 = by the lengths of the runs, 3 and 4 = as 1
// and 2 with the bits of uneven streams, 5 = the latest positions of the contexts, else the sets of lags in pieces of `way` steps (a multiple of 32)
extern "C" int rosa_host_batch(uint32_t way, const uint32_t* q, const uint32_t* k, const uint32_t* v, size_t n_streams,
                               uint32_t T, uint32_t* out) {
    const size_t wps = (T + 31u) / 32u;
    for (size_t s = 0; s < n_streams; ++s) {
        const size_t at = s * wps;
        if (way <= 4u) by_contexts(q + at, k + at, v + at, T, way > 2u ? context::bits_for_uneven(T) : context::bits_for(T), way == 2u || way == 4u, way == 0u, out + at);
        else if (way == 5u) {
            const uint32_t half = (uint32_t)wps / 2u;   // in two pieces
            if (half) by_heads(q + at, k + at, v + at, 32u * half, 0u, out + at);
            by_heads(q + at, k + at, v + at, T, half, out + at);
        } else if (!by_lags(q + at, k + at, v + at, T, way, out + at)) return 1;
    }
    return 0;
}

// The rows of each of the pieces that a stream of T steps is cut into where `wanted` are; returns how many there are.
extern "C" uint32_t rosa_host_pieces(uint32_t T, uint32_t wanted, uint32_t* row0, uint32_t* row1) {
    const uint32_t words = (T + 31u) / 32u, pieces = heads::pieces_with_rows(words, wanted), rows = heads::rows_of_piece(words, pieces);
    for (uint32_t i = 0; i < pieces; ++i) {
        row0[i] = i * rows < words ? i * rows : words;
        row1[i] = row0[i] + rows < words ? row0[i] + rows : words;
    }
    return pieces;
}

// What the warp of a piece asks before it puts any key in: whether the runs of the first `rows` rows alone make its walks too long.
extern "C" int rosa_host_runs_too_long(const uint32_t* q, const uint32_t* k, uint32_t rows, uint32_t most) {
    uint32_t keys[2] = {0, 0}, in[2] = {0, 0};
    for (uint32_t w = 0; w < rows; ++w)
        for (uint32_t z = 0; z < 2u; ++z) {
            keys[z] += (uint32_t)__builtin_popcount(heads::ends_of_runs(z ? ~k[w] : k[w]));
            in[z] += heads::ends_of_runs(z ? ~q[w] : q[w]) != 0u;
        }
    return heads::walks_too_long(keys[0], in[0], most) || heads::walks_too_long(keys[1], in[1], most);
}
