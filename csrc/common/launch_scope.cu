// Programmatic dependent launch for the launches of the calling thread (launch.cuh).
#include "launch.cuh"

// Returns the previous setting.
extern "C" int z2h_pdl_scope(int on) {
  const int before = z2h::pdl_scope;
  z2h::pdl_scope = on;
  return before;
}
