/*
 * lanes_harness.cpp -- TEST INFRASTRUCTURE.  Which lanes of a warp take which branch, computed on the CPU
 * with the functions that the kernels call.
 */
#include "../cuteflow_gb300/csrc/cf_flux.h"

using namespace cf;

/* The edge kernel's shape in a recording forward of a context with the given shape */
extern "C" void harness_recording_shape(int32_t eblock, int32_t ept, int32_t chosen, int32_t* out) {
  StepArgs a;
  std::memset(&a, 0, sizeof(a));
  a.eblock = eblock;
  a.ept = ept;
  recording_shape(a, chosen != 0);
  out[0] = a.eblock;
  out[1] = a.ept;
}

/* The dispatch rules on a device of sms SMs */
extern "C" int harness_edge_block(long long ne_pad, int32_t sms) { return first_edge_block(ne_pad, sms); }
extern "C" int harness_adj_blocks(int32_t n_etiles, int32_t sms) { return adj_hllc_blocks(n_etiles, sms); }
extern "C" int harness_two_lanes(int32_t n_ctiles, int32_t sms) {
  StepArgs a;
  std::memset(&a, 0, sizeof(a));
  a.n_ctiles = n_ctiles;
  a.sms = sms;
  return two_lanes(a);
}

/* The warps of the list kernel over both phases of a part (16 edges each, two lanes an edge): how many hold
 * edges of both arithmetic types under the tuning mask, by the kernel's rule, and by the edges' numbers. */
extern "C" int harness_list_warps(const cf_mesh* m, const cf_params* p, const int32_t* elem_class, int32_t mask,
                                  int32_t* warps, int32_t* mixed, int32_t* mixed_by_number) {
  Prep P;
  std::string err;
  const int rc = prepare_mesh(m, p, P, err, elem_class);
  if (rc != CF_OK) return rc;
  *warps = *mixed = *mixed_by_number = 0;
  for (const auto* list : {&P.elist1, &P.elist2}) {
    const int n = (int)list->size();
    for (int w = 0; w < n; w += 16) {
      int rule = 0, number = 0;
      for (int i = w; i < n && i < w + 16; ++i) {
        rule |= 1 << int_products(mask, i);
        number |= 1 << int_products(mask, (*list)[i]);
      }
      ++*warps;
      *mixed += rule == 3;
      *mixed_by_number += number == 3;
    }
  }
  return 0;
}
