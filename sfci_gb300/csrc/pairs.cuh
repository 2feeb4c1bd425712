// Terms between two given sets of determinants: entry points of pairs.cu.
#pragma once

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

// Adds every term of (H - lambda) v that lands on a key of the open-addressing
// table (`slots` slots, empty ones key_empty) to that slot's accumulators (split
// form, see common.cuh).  *done false: declined as above (but for repeated keys,
// whose terms are added like any others); the accumulators may then hold a part of
// the sums.
template <int W>
int pairs_project(Ctx& c, const typename KeyOf<W>::T* keys, const double* amps, u64 n, double lambda,
                  const typename KeyOf<W>::T* table, u64 slots, u64* plo, u64* phi, bool* done);

}  // namespace sfci
