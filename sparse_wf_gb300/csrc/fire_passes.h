// fire_passes.h -- how many walkers a pass of the local energy takes (host arithmetic only).
#pragma once

namespace fire {

// Rounds that the elimination of `mats` matrices per walker takes over `walkers` walkers in passes of c, `places` matrices on
// the GPU at once.
inline long elimination_rounds(long walkers, long c, int mats, int places) {
  auto rounds = [&](long w) { return (w * mats + places - 1) / places; };
  return walkers / c * rounds(c) + rounds(walkers % c);
}

// Walkers per pass, c at most: reduced to whole rounds of the elimination where the batch then takes fewer of them, one for
// every pass that this adds at least.  512 walkers of 322 electrons (304 places): passes of 153 take 4 passes and 10 rounds,
// passes of 152 4 and 7.  A batch that fits one pass stays whole: splitting it saves no round (100 walkers take two either
// way, in 127.2 ms as one pass, in 131.6 as 76 + 24; 153 take three, 174.4 and 178.3).
inline int pass_walkers(long walkers, int c, int mats, int places) {
  const int round = mats > 0 ? places / mats : 0;  // walkers of a round
  if (round < 1 || c <= round || c >= walkers) return c;
  const int d = c - c % round;
  const long saved = elimination_rounds(walkers, c, mats, places) - elimination_rounds(walkers, d, mats, places);
  const long added = (walkers + d - 1) / d - (walkers + c - 1) / c;
  return saved > 0 && saved >= added ? d : c;
}

}  // namespace fire
