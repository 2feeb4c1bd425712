// Row-driven product: entry point of rows.cu.
#pragma once

#include "common.cuh"
#include "internal.h"

namespace sfci {

// What a row-driven product leaves behind for the final selection.
template <int W>
struct RowsResult {
  typename KeyOf<W>::T* sk = nullptr;  // survivors of the cut, any order
  double* sa = nullptr;
  u64 nsurv = 0;
  u64 uniq = 0;      // merged distinct determinants
  u64 terms = 0;     // generated terms
  u64 dexact[2] = {0, 0};  // <v|Hv>, exact 128-bit fixed point
  u64 units = 0;     // work units
  u64 rounds = 1;       // fillings of the survivor buffer
  bool pruned = false;  // survivors were cut to the output capacity on the way
};

// The product's terms generated and merged row by row (see rows.cu), with nx extra
// sources after the ns determinants of one term each (key, amplitude).  *done is
// false when the input is outside what the row form handles (the caller then
// runs the partitioned pipeline): mixed spin counts, more rows or pairs than
// its tables take, too little device memory, or a term too large for its
// accumulators.
template <int W>
int rows_product(Ctx& c, const typename KeyOf<W>::T* keys, const double* amps, u64 ns, u64 nx, double lambda,
                 double coeff, u64 cap, RowsResult<W>* out, bool* done);

// device memory of the row form's per-context tables
void rows_free(Ctx& c);

}  // namespace sfci
