// A cuFFT call that fails, for tests/test_batch_serving.py: replaces the plan of a
// handle's forward transform by a handle that cuFFT does not know (it answers
// CUFFT_INVALID_PLAN on the host) and returns the one that was there.
#include "internal.h"

extern "C" int swap_forward_plan(npme_handle *h, int plan) {
  const cufftHandle old = h->pf->plan;
  h->pf->plan = (cufftHandle)plan;
  return (int)old;
}
