// dispatch.cpp -- which kernel a launch of the plain FP64 form goes to, asked
// of the library's own rules (hyc_internal.h) on this machine's device.
// Arguments, five a launch: scheme ii jj layers fields, and for all of them
// first "free" or the tile shape that a caller fixed, as 32x16.  A line each:
// "strip", or "tile TXxTY tma" / "tile TXxTY plain".
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "hyc_args.h"
#include "hyc_internal.h"

int main(int argc, char **argv) {
  hyc::TileShape s{32, 16};
  const bool fixed = sscanf(argv[1], "%dx%d", &s.tx, &s.ty) == 2;
  for (int q = 2; q + 4 < argc; q += 5) {
    hyc::TileArgs a;
    memset(&a, 0, sizeof a);
    const int scheme = atoi(argv[q]), layers = atoi(argv[q + 3]);
    a.ii = atoi(argv[q + 1]);
    a.jj = atoi(argv[q + 2]);
    a.nfld = atoi(argv[q + 4]);
    const hyc::TilePlan p = hyc::tile_plan(scheme, a, layers, s, fixed);
    if (p.strip) puts("strip");
    else printf("tile %dx%d %s\n", p.shape.tx, p.shape.ty, p.tma ? "tma" : "plain");
  }
  return 0;
}
