// How many CTAs a work slot gets (host arithmetic only).
#pragma once

namespace negf {

// A launch with fewer slots than half the SMs leaves the others idle, so each slot gets a cluster of
// 2, 4 or 8 CTAs while all slots still run at once (fit(c): clusters of c that fit the GPU together) and
// an n x n product has a 32 x 64 output piece for every CTA.
template <class Fit>
inline int team_rule(int n, int slots, int sms, Fit fit) {
  if (n <= 32) return 1;
  const int pieces = ((n + 31) / 32) * ((n + 63) / 64);
  for (int cl = 8; cl > 1; cl /= 2)
    if (cl <= pieces && slots * cl <= sms && fit(cl) >= slots) return cl;
  return 1;
}

// The size that the rule sees for a decimation of leads of up to n: a step's largest product is 2n x 2n, but
// below 49 the panels that every CTA repeats and the cluster's barriers cost more than the products gain.
// 18 energies, one CTA each -> clusters: n = 24 1.04 -> 1.30 ms, 32 1.11 -> 1.37, 48 2.58 -> 2.68,
// 52 3.36 -> 3.14, 64 3.76 -> 3.42.
inline int ls_team_n(int n) { return n > 48 ? 2 * n : 1; }

}  // namespace negf
