// Which form of attention a round takes, and how the decode form cuts contexts: plain arithmetic on sizes, no device.
#pragma once

namespace lcu {

// ---- the decode form (attention.cu): CTAs of `tiles` tiles of 64 positions, `splits` of them for the longest context of the round.
// Planned for the round's own contexts, rounded up to `max_tiles` = 2^n tiles so that a captured round stays valid while they grow,
// and not for the longest that the cache allows (8B shape, 16 sequences of 100 to 290 tokens: 3.88 -> 3.71 ms per round).
struct AttnPlan {
    int splits, tiles;
};
// What decides, measured per layer with 1 to 64 sequences of 100 to 3950 tokens, 1 to 32 KV heads, heads of 64 and 128:
//   - enough CTAs to fill the GPU about four times over, no more: eight times is up to 45 % slower where contexts are long (16 sequences
//     of 3900 tokens, one KV head: 82 -> 119 us), since a merge costs 2 us with 2 splits, 6 with 8, 15 with 16 and 60 with 62;
//   - hence at least two tiles a CTA from 9 tiles on (one sequence of 900 tokens: 26.7 -> 24.7 us), three from 33 on (one of 3900:
//     37.5 -> 33.3 us), and fewer CTAs in all where there are many splits;
//   - a single CTA where the merge through scratch costs more than its tiles: up to two, and with heads of 64 (0.8 us a tile instead
//     of 1.5) up to four once the heads alone are a wave's quarter (1B shape, 8 sequences of 180 tokens: 40.8 -> 39.2 us).
// `clusters`: the splits of a token merge inside a thread-block cluster where it has room for them (rounds of one and two tokens).
inline AttnPlan attn_plan(int nkvh, int dh, int n_tok, int max_tiles, int sms, bool clusters) {
    const long ctas = (long)nkvh * n_tok;
    if (ctas >= 8L * sms || max_tiles <= 1) return {1, max_tiles};
    if (!clusters && (max_tiles <= 2 || (dh == 64 && max_tiles <= 4 && 4 * ctas >= sms))) return {1, max_tiles};
    const long slots = (long)sms * (max_tiles <= 16 ? 4 : max_tiles <= 32 ? 3 : 2);
    int t = (int)((ctas * max_tiles + slots - 1) / slots);
    const int least = max_tiles > 32 ? 3 : max_tiles > 8 ? 2 : 1;
    t = t > 4 ? 4 : t < least ? least : t;
    int z = (max_tiles + t - 1) / t;
    int z_cap = 2048 / n_tok;  // bounds the partial-output scratch
    z_cap = z_cap > 64 ? 64 : z_cap < 1 ? 1 : z_cap;
    if (z > z_cap) {
        z = z_cap;
        t = (max_tiles + z - 1) / z;
    }
    return {z, t};
}

// ---- rounds that hold prompts
enum AttnForm {
    ATTN_SPLIT,    // the decode form, a token at a time
    ATTN_ROWS64,   // mma.sync, 64 query rows a CTA (attn_prefill_kernel)
    ATTN_ROWS256,  // tcgen05, 256 query rows a CTA (attn_tc_kernel)
};
// Cost of a form in us per layer: the slowest CTA, or all CTAs' work on the SMs if that is longer (constants by heads of 64 and 128,
// fitted to 492 rounds: 1 to 61 sequences, prompts of 2 to 1000 tokens behind 0 to 1900 cached ones, 1 to 8 query heads per KV head; the
// choice is never more than 4 % off the better form).  A CTA of 256 rows pays for all of them: where a
// round is mostly decoded tokens with few rows each, the smaller one wins until contexts are long (60 sequences of 32 heads: up to
// 250 positions with heads of 128, 1200 with heads of 64).
struct AttnCost {
    double start, tile, two, chain_start, chain_tile;  // us of an SM per CTA and per tile (of two row tiles); the slowest CTA's
};
template <class Req>  // with `pos` cached tokens and `len` new ones
double attn_form_cost(AttnForm form, int dh, int group, int nkvh, const Req *reqs, int n_req, int sms) {
    static const AttnCost rows64[2] = {{2.3, 0.7, 0.7, 0.4, 1.65}, {1.8, 1.4, 1.4, 0.0, 1.85}};
    static const AttnCost rows256[2] = {{5.9, 0.8, 2.0, 2.9, 1.2}, {4.2, 1.5, 2.5, 0.8, 1.55}};
    const bool big = form == ATTN_ROWS256;
    const AttnCost &c = (big ? rows256 : rows64)[dh == 64 ? 0 : 1];
    const long per = (big ? 256 : 64) / group, tile = big ? 128 : 64;
    double work = 0., slowest = 0.;
    for (int i = 0; i < n_req; ++i) {
        const long pos = (long)reqs[i].pos, len = (long)reqs[i].len;
        if (form == ATTN_SPLIT) {  // tiles of 64 positions for every token
            work += (double)len * ((double)pos + 0.5 * (double)len + 64.) / 64. * (dh == 64 ? 0.42 : 0.75);
            continue;
        }
        for (long j = 0; j < len; j += per) {
            const long rows = len - j < per ? len - j : per, tiles = (pos + j + rows + tile - 1) / tile;
            const bool two = big && rows * group > 128;
            work += c.start + (two ? c.two : c.tile) * (double)tiles;
            const double chain = c.chain_start + (two && c.two > c.chain_tile ? c.two : c.chain_tile) * (double)tiles;
            if (chain > slowest) slowest = chain;
        }
    }
    work *= (double)nkvh / sms;
    return form == ATTN_SPLIT ? 10. + work : work > slowest ? work : slowest;
}
// rows64, rows256: whether the form is possible.  Where the 64-row form is not (its page table is held in shared memory), the other
// choice for a few tokens behind a long context is the decode form: it cuts the context (16 tokens behind 60000: 0.66 instead of 0.84 ms).
template <class Req>
AttnForm attn_form(int dh, int group, int nkvh, const Req *reqs, int n_req, int sms, bool rows64, bool rows256) {
    const AttnForm other = rows64 ? ATTN_ROWS64 : ATTN_SPLIT;
    if (!rows256) return other;
    return attn_form_cost(ATTN_ROWS256, dh, group, nkvh, reqs, n_req, sms) < attn_form_cost(other, dh, group, nkvh, reqs, n_req, sms) ? ATTN_ROWS256 : other;
}

}  // namespace lcu
