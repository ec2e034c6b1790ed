// pmproduct.h -- short products of polynomial matrices (pmproduct.cu).
#pragma once
#include "rr_internal.h"

namespace rr {

// C[i][j][t - lo], t in [lo, lo + cnt), of A (m x r, la coefficients) times B
// (r x k, lb coefficients) mod p for nb generators; entry (i, j) of generator z
// starts at X + z x_bs + i x_rs + j x_cs.
struct DirectProduct {
  const uint32_t* A;
  int64_t a_rs, a_cs, a_bs;
  int m, r, la;
  const uint32_t* B;
  int64_t b_rs, b_cs, b_bs;
  int k, lb;
  uint32_t* C;
  int64_t c_rs, c_cs, c_bs;
  int lo, cnt;
  ModP M;
  // set by direct_product: 2^32, 2^40, 2^48 mod p, R^2 mod p, shared-memory offset
  uint32_t w[3], r2;
  int red_off;
};

int direct_product_max(int r);   // largest la - 1
int direct_product_prepare();
int direct_product(DirectProduct P, int nb, cudaStream_t s);

}  // namespace rr
