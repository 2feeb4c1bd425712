// Terms between two given sets of determinants: entry points of pairs.cu.
#pragma once

#include <cmath>

#include "common.cuh"
#include "internal.h"

namespace sfci {

// <psi|H|psi> over psi's own support; *terms: the terms of H psi; *links: pairs of
// alpha strings one or two moves apart.  *done false: declined (mixed spin counts,
// repeated keys, more strings than the rank tables take, no memory or none within the
// device budget, a term out of range), nothing computed.
template <int W>
int pairs_energy(Ctx& c, const typename KeyOf<W>::T* keys, const double* amps, u64 n, double* E, u64* terms,
                 u64* links, bool* done);

// Where the search pays for a projection of T terms onto a table of `slots` slots,
// RA strings of a spin: the sweep takes about 25 ps a term, the search 1.75 ns a slot
// (every slot is ranked and listed) besides a part that grows with the rank tables.
// Measured, us of the linear product with the search and with the sweep: 28 orbitals,
// 64 sources onto 1,000 determinants 855 / 751, onto 1,000,000 5547 / 2074; 1,000
// onto 1,000 1984 / 3266, onto 100,000 2632 / 2647, onto 1,000,000 6185 / 3257; 4,000
// onto 1,000 4197 / 10503, onto 1,000,000 8690 / 8817; 34 orbitals, 256 onto 1,000
// 2323 / 2501, 1,000 onto 10,000 5967 / 6369; 10 orbitals, 4,000 onto 1,000 664 / 768,
// onto 10,000 755 / 718.
inline bool pairs_project_pays(u64 T, u64 slots, u64 RA) {
  return (double)T >= 3e6 + 70.0 * (double)slots + 4000.0 * std::sqrt((double)RA);
}

// Adds every term of (H - lambda) v that lands on a key of the open-addressing
// table (`slots` slots, empty ones key_empty) to that slot's accumulators (split
// form, see common.cuh).  T: the most terms v can have.  *done false: declined where
// the sweep is faster, or as above (but for repeated keys,
// whose terms are added like any others); the accumulators may then hold a part of
// the sums.
template <int W>
int pairs_project(Ctx& c, const typename KeyOf<W>::T* keys, const double* amps, u64 n, u64 T, double lambda,
                  const typename KeyOf<W>::T* table, u64 slots, u64* plo, u64* phi, bool* done);

}  // namespace sfci
