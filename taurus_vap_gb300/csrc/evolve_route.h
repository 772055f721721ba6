// The two routes of the Thouless evolution and what each finds ready (host
// code; tests/evolve_route_check.cpp).
#pragma once

#include "tvap.h"

namespace tvap {

// products(): S = 1 + Z^T Z, A1 = U0 + V0 Z and A2 = V0 + U0 Z into the work
// memory; coop(): the cooperative launch, which forms them itself where
// coop_forms says so, TVAP_ERR_ARG where it does not run (n, shared memory or
// co-resident grid); single(): the single-CTA inverse and the products with
// it, which need them.
template <class Products, class Coop, class Single>
int evolve_route(bool coop_forms, Products products, Coop coop, Single single) {
  int rc = TVAP_OK;
  if (!coop_forms && (rc = products())) return rc;
  if ((rc = coop()) != TVAP_ERR_ARG) return rc;
  if (coop_forms && (rc = products())) return rc;
  return single();
}

}  // namespace tvap
