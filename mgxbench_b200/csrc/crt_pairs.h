// crt_pairs.h -- when the CRT form's residue products run on pairs of CTAs, and on how many.  By itself, so that
// the CPU tests compile it too.
#pragma once

namespace mgx {
namespace crt {

// Pairs for a product of `items` work items of single CTAs, `pairs` of pairs, on `sms` SMs that can hold
// `clusters` pairs at once; 0: CTAs alone.  Pairs where their rounds of items are no more than single CTAs' (an
// odd last tile row makes half a pair idle) and four rounds or more pay for the pairs' setup: 1333 x 2011 x
// 1777, 5 rounds, 143 us against 147 alone; 1024^3, 2 rounds, 62.9 against 62.5.
inline int pairs_to_launch(long long items, long long pairs, int sms, int clusters)
{
    const int slots = clusters < sms / 2 ? clusters : sms / 2;
    if (slots <= 0 || pairs < 4ll * slots) return 0;
    return (pairs + slots - 1) / slots <= (items + sms - 1) / sms ? slots : 0;
}

}  // namespace crt
}  // namespace mgx
