// pmleaf.h -- one block of leaves of the PM-basis (pmleaf.cu).
#pragma once
#include "rr_internal.h"

namespace rr {

// K order-1 leaves on the first K coefficients of G (m = 2n rows, n <= 32
// columns) for nb generators; generator z starts at G + z g_bs, delta + z m and
// Mout + z out_bs.
struct LeafBlock {
  const uint32_t* G;      // G[i][c][t]: row stride g_rs, column stride g_cs, t < K
  int64_t g_rs, g_cs, g_bs;
  int m, n, K;
  int64_t* delta;         // [m], in/out
  uint32_t* Mout;         // Mout[i][j][t], t <= K
  int64_t out_rs, out_cs, out_bs;
  ModP M;
  int* status;            // 2: a zero row scale; 3: a wait gave up
  uint64_t wait_ns;       // a wait gives up after this long
  int missing;            // words the first hand-off expects beyond those that come (0; checks of the give-up path)
  // set by leaf_block_launch
  int nres, nbas;         // residual and basis CTAs of a cluster
  uint32_t two16;         // 2^16
};

int leaf_block_max(int m);        // largest K
int leaf_block_prepare(int n);    // shared-memory limit of the variant for n columns
int leaf_block_launch(LeafBlock P, int nb, cudaStream_t s);

}  // namespace rr
