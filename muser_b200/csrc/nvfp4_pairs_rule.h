// When the NVFP4 GEMM takes pairs of SMs: plain C++, so that a host program can hold the rule against measurements
// (tests/test_pairs_rule_cpu.py).
#pragma once
#include <stdint.h>

namespace muser {

enum class PairForm { plain, group, fused }; // single outputs, projections in one launch, the SwiGLU forms

// Pairs of SMs or single CTAs for `n_tiles` weight-row tiles of `tokens` tokens and `slabs` 256-value steps each, on a device of
// `sms` SMs that holds `room` pairs at once?  The same bits either way.
//
// Many tiles: a round of pairs takes 0.86 to 0.93 of a round of single CTAs (us, single / pairs at 2048 tokens: 5120 x 5120
// 32.3 / 27.7, 7168 x 5120 in a group 37.7 / 32.4, 5120 x 27648 138 / 120, gate/up 237 / 220), but an odd block of 128 tokens is
// half of a pair's tile (gate/up at 384 tokens, five rounds against six: 55 / 60).
//
// One round: a slab takes a pair 0.28 us and a single CTA 0.35, and a pair starts 0.3 us later, a group of them 0.7.  Few
// tokens leave the second CTA of a pair without any, and the single form fetches their rows only; and a launch that leaves SMs
// free lets the next one set up and load beside it, which twice the CTAs do not.  us, single / pairs / tiles, weights from HBM:
//   plain, 16 tokens     4 slabs 4.5 / 4.8 at 8, 4.9 / 7.1 at 74; 11 slabs 7.3 / 7.2 at 16, 7.6 / 7.7 at 28, 8.2 / 8.9 at 40
//          64            4 slabs 5.4 / 5.3 at 28, 6.0 / 7.2 at 74; 11 slabs 7.8 / 7.4 at 16, 10.5 / 10.4 at 74
//          128           4 slabs 6.4 / 5.7 at 28, 6.5 / 7.7 at 74; 11 slabs 9.2 / 8.2 at 28, 11.5 / 10.2 at 74
//   gate/up, 16          4 slabs 7.5 / 7.9 at 16, 7.4 / 9.9 at 74; 20 slabs 13.1 / 12.7 at 16, 14.1 / 18.0 at 40, 16.5 / 17.9 at 74
//            128         4 slabs 7.7 / 8.1 at 16; 20 slabs 13.4 / 12.8 at 16, 14.4 / 14.8 at 40, 16.9 / 16.0 at 74
//   group, single over pairs: at 64 tokens 0.91 to 0.99 up to 11 slabs, 1.02 to 1.07 with 20; at 128 up to 37 tiles 1.01 to 1.12,
//            with 74 tiles 0.78 to 0.93; at 384 with 74 tiles 0.91 (5 slabs); at 512 with 37 tiles 0.90 (4), 0.97 (11), 1.01 (20)
//   long rows: 32 slabs, plain at 32 and 48 tokens 18.4 / 16.9 at 56; SwiGLU of 108 slabs at 16 tokens 43.7 / 38.1 at 20, 54.6 /
//            49.2 at 56; a group of 32 slabs and 72 tiles at 128 tokens 20.5 / 18.7
// Over 4000 points (4 to 108 slabs, 4 to 108 tiles, 1 to 1000 tokens, the three forms) the choice took 1.002 times the faster
// form's time on average and 1.1 times at worst, calls that cut K aside.
inline bool pairs_pay(uint32_t sms, uint32_t room, uint32_t n_tiles, uint32_t tokens, uint32_t slabs, PairForm form) {
    if (!room) return false;
    const uint64_t blocks = ((uint64_t)tokens + 127) / 128, pair_tiles = n_tiles * ((blocks + 1) / 2);
    const uint64_t pair_rounds = (pair_tiles + room - 1) / room, single_rounds = (n_tiles * blocks + sms - 1) / sms;
    if (pair_rounds * 9 > single_rounds * 10) return false;
    const auto of_sms = [&](uint32_t part) { return pair_tiles * part > sms; }; // more tiles than such a part of the SMs
    const bool crowded = pair_rounds == 1 && of_sms(form == PairForm::fused ? 5 : 4); // little is left for the next launch
    const bool odd = blocks % 2, wasted = odd && blocks > 1 && pair_rounds == single_rounds; // an odd block's pairs gain no round
    switch (form) {
    case PairForm::plain:
        if (tokens < 64 && (slabs < 9 || (of_sms(tokens < 40 ? 8 : 4) && slabs < (tokens < 32 ? ~0u : tokens < 40 ? 30u : 24u)))) return false;
        return !crowded || !odd || slabs >= (tokens < 96 ? 14 : tokens < 112 ? 10 : 7 * pair_tiles > 2 * sms ? 8 : 0);
    case PairForm::group:
        if (tokens < 112 && (slabs < (tokens < 96 ? 16 : 11) || (of_sms(tokens < 64 ? 8 : 4) && slabs < (tokens < 96 ? ~0u : 24u)))) return false;
        if (crowded && blocks == 1) return slabs >= 24 || (slabs >= 10 && 8 * pair_tiles <= 3 * sms);
        return crowded ? slabs >= (odd ? 16 : 10) : slabs >= (wasted && pair_rounds > 1 ? 9 : 0);
    case PairForm::fused:
        if (tokens < 64 && of_sms(tokens >= 48 ? 5 : slabs < 16 ? 8 : slabs < 40 || tokens < 8 ? 6 : 4) &&
            slabs < (tokens < 16 ? ~0u : tokens < 32 ? 80u : tokens < 48 ? 40u : 24u)) return false;
        return slabs >= (crowded ? 20 : wasted ? 16 : 12);
    }
    return false;
}

} // namespace muser
