// batch.cpp -- cnuity's layers per launch, asked of the library: pairs of
// arguments "cells layers", a line each.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>

#include "hyc_internal.h"

int main(int argc, char **argv) {
  for (int q = 1; q + 1 < argc; q += 2) printf("%d\n", hyc::cnuity_batch(atoll(argv[q]), atoi(argv[q + 1])));
  return 0;
}
