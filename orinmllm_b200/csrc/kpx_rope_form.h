// Which form of the RoPE kernel a call takes.  Host code only.
#pragma once
#include <stdint.h>

namespace kpx {

enum class RopeForm {
  kFlat,         // a thread per rotation pair-group, tables and weights fetched where they are used
  kEarlyTables,  // the same, fetched four floats at a time before the norm
  kOneToken,     // a CTA per token, what its heads share in shared memory
  kTwoTokens,    // a CTA per two tokens
};

struct RopeCall {
  int elt_bytes, head_size;
  int64_t tokens;
  bool norm, aligned;           // aligned: tables and weights lie on 16-byte boundaries
  int64_t ctas;                 // of the flat forms, a thread per item
  int64_t flat_fit, early_fit;  // CTAs of either that the device holds at a time
};

// From kRowsFrom tokens on 16-bit rows of 128 take rope_rows_kernel (256 tokens: 4.4 / 2.8 us with / without a norm
// against 3.9 / 2.7 of the flat forms; 512: 5.0 / 3.1 against 5.3 / 3.8), from kRowsPairs on with two tokens a CTA
// (777: 7.0 / 4.4 against 6.2 / 3.9 with one; 2048: 10.4 / 6.3 against 11.5 / 7.3).
constexpr int64_t kRowsFrom = 400, kRowsPairs = 1400;

// Tables fetched early shorten the chain of a call with a norm (without one there is no more to fetch than the chain
// brings anyway: bf16 28/4, 1 and 64 tokens 1.89 / 2.14 us early, 1.81 / 2.06 flat) and cost registers: an SM holds
// fewer CTAs (16-bit rows 3 for 5, fp32 4 for 6).  So that form is for calls that it holds at once, and beyond what the
// other holds at once for those that it takes one round more for at most; heads wider than 128 gain more by it and
// take it in any case.  A sixteenth of a round more costs next to nothing
// (heads of 64, 32/8, 2048 tokens, 1792 CTAs, four early rounds and 16 CTAs: 8.0 us early, 8.5 flat, alone).
// norm + RoPE + append and a decode launch of 64 short sequences, us, flat / early: fp16 32/8 heads of 128, 256 tokens
// (448 CTAs) 15.3 / 14.6, 320 (560) 15.4 / 15.9; 64/8, 256 (704) 16.2 / 16.7, 320 (880) 18.4 / 16.7; heads of 64, 32/8,
// 800 (700) 14.8 / 15.5, 1600 (1400) 17.3 / 18.4; fp32 32/8, 160 (560) 15.0 / 13.9, 224 (784) 15.1 / 15.6, 320 (1120)
// 17.1 / 15.8; heads of 256, bf16 28/4, 256 (640) 14.5 / 14.3, 900 (2250) 26.0 / 21.8, 8000 151 / 116, fp16 12/2, 600 (675) 11.7 /
// 11.9, fp32 32/8, 8000 213 / 206.
inline RopeForm rope_form(const RopeCall& c) {
  if (c.elt_bytes == 2 && c.head_size == 128 && c.tokens >= kRowsFrom)
    return c.tokens < kRowsPairs ? RopeForm::kOneToken : RopeForm::kTwoTokens;
  if (!c.norm || !c.aligned) return RopeForm::kFlat;
  auto rounds = [&](int64_t fit) { return (c.ctas + fit - 1 - fit / 16) / fit; };
  const int64_t early = rounds(c.early_fit), flat = rounds(c.flat_fit);
  if (early <= 1 || c.head_size > 128) return RopeForm::kEarlyTables;
  return flat > 1 && early <= flat + 1 ? RopeForm::kEarlyTables : RopeForm::kFlat;
}

}  // namespace kpx
