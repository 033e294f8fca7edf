// How many groups of 16 columns of the state a block of the chunked recurrences' walk takes (chunked_recurrence.cu): 1 (eight warps share them), 2
// or 4 (chunk_wide_kernel). Plain C++, so that a host compiler takes it too.
//
// The cheapest of: rounds of blocks the GPU needs, times how long a step of 32 tokens takes with that many columns (hundredths of a microsecond).
// Blocks are counted as if every request were as long as the longest: a step of one long request beside short ones is one chain, and
// the short ones' blocks run on the SMs it leaves. Counted by requests, a request of 2,048 tokens beside fifteen of 97 (8 heads, a decay alone)
// walked 64 columns a block: 276 us against 158.
// Both sides measured, a whole recurrence, 16 heads, us (16 columns a block | 32 | 64): states of 128 x 128 with a decay alone, one request of 2,048
// tokens 157 | 199 | 281, with another of 97 160 | 202 | 281, with fifteen of 97 302 | 246 | 323, two of 1,024 161 | 132 | 173, four of 512 165 | 135 | 120, eight of
// 256 161 | 141 | 126; with the delta rule one of 2,048 208 | 258, with one of 97 209 | 264, four of 512 215 | 182; 64 x 64 with the delta rule, one of 2,048
// 160 | 180, eight of 256 121 | 102; with a decay alone (two blocks an SM, which slow one another down) one of 2,048 121 | 130, two of 1,024 83 | 88, four of 512
// 72 | 66, eight of 256 74 | 63.
#pragma once

namespace sb {

struct WalkStep { int alone, paired; };      // us / 100 a step: one block an SM; two at a time there (0: one block fills an SM)

// big: states of more than 64 rows. cols: groups of 16 columns. chunks: of all listed requests, longest: of the longest of them.
inline int walk_groups(bool delta, bool big, long long heads, long long cols, long long chunks, long long longest, long long sms) {
  const WalkStep one = delta ? WalkStep{big ? 187 : 154, 0} : big ? WalkStep{157, 0} : WalkStep{133, 205};
  const WalkStep two = delta ? WalkStep{big ? 260 : 185, 0} : big ? WalkStep{213, 0} : WalkStep{160, 285};
  const WalkStep four = WalkStep{342, 0};
  if (longest < 1) longest = 1;
  auto cost = [&](long long groups, WalkStep s) {
    const long long blocks = (chunks * heads * ((cols + groups - 1) / groups) + longest - 1) / longest;
    const bool paired = s.paired > 0 && blocks > sms;
    const long long at_once = paired ? 2 * sms : sms;
    return (blocks + at_once - 1) / at_once * (paired ? s.paired : s.alone);
  };
  const long long c1 = cost(1, one), c2 = cost(2, two);
  if (big && !delta) {
    const long long c4 = cost(4, four);
    if (c4 < c1 && c4 < c2) return 4;
  }
  return c2 < c1 ? 2 : 1;
}

}  // namespace sb
