// Every route of the evolution, and every failure on it: whoever reads S and A finds them formed by this call, and once.
#include <cstdio>
#include <initializer_list>

#include "evolve_route.h"

using namespace tvap;

int main() {
  int bad = 0;
  const int codes[] = {TVAP_OK, TVAP_ERR_ARG, TVAP_ERR_CUDA};
  for (int forms = 0; forms < 2; ++forms)
    for (int rc_products : {TVAP_OK, TVAP_ERR_CUDA})
      for (int rc_coop : codes)
        for (int rc_single : {TVAP_OK, TVAP_ERR_CUDA}) {
          int products = 0, coop = 0, single = 0;
          const int rc = evolve_route(
              forms != 0, [&]() { return ++products, rc_products; },
              [&]() {
                bad += products != (forms ? 0 : 1);
                return ++coop, rc_coop;
              },
              [&]() {
                bad += products != 1;
                return ++single, rc_single;
              });
          const bool first = !forms && rc_products != TVAP_OK;
          bad += coop != (first ? 0 : 1);
          const int expect = first                      ? rc_products
                             : rc_coop != TVAP_ERR_ARG  ? rc_coop
                             : rc_products != TVAP_OK   ? rc_products
                                                        : rc_single;
          bad += rc != expect;
          bad += single != (!first && rc_coop == TVAP_ERR_ARG && rc_products == TVAP_OK ? 1 : 0);
        }
  std::printf("bad %d\n", bad);
  return bad != 0;
}
