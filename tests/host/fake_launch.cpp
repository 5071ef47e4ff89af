// fake_launch.cpp -- stand-ins for the launchers that hyc_ens_host.cpp calls:
// each names the device pointers its kernel reads and writes (fake_cuda.h).
#include <cuda_runtime.h>

#include "hyc_args.h"
#include "hyc_ens.h"
#include "hyc_internal.h"
#include "hyc_tmap.h"

#include "fake_cuda.h"
#include "fake_launch.h"

int fake_fail_launches = 0, fake_step_launches = 0, fake_maps = 0;
bool fake_strip = true;

static bool step_launch() {  // counted; false where it is to fail
  fake_step_launches++;
  return !(fake_fail_launches > 0 && --fake_fail_launches == 0);
}

namespace hyc {

bool tmap_available() { return true; }
bool tmap_encode3(CUtensorMap *, const void *, int, long long, long long, long long, long long, long long, int, int) {
  fake_maps++;
  return true;
}
void set_library_error(const char *) {}
bool march_takes(int, const TileArgs &, int) { return fake_strip; }
cudaError_t launch_xctilr(double *a, long long, int, int, int, int, int, int, int, int, cudaStream_t s) {
  fake::use(a, s);
  return cudaSuccess;
}
cudaError_t launch_march_queue(int, const TileArgs *basins, const int4 *items, int, int *head, int, cudaStream_t s) {
  if (!step_launch()) return cudaErrorInvalidValue;
  for (const void *p : {(const void *)basins, (const void *)items, (const void *)head}) fake::use(p, s);
  return cudaSuccess;
}
cudaError_t launch_mix_col2(int, const MixBasin *basins, const int4 *items, int, int *head, int, int, bool, bool, int *err,
                            cudaStream_t s) {
  if (!step_launch()) return cudaErrorInvalidValue;
  for (const void *p : {(const void *)basins, (const void *)items, (const void *)head, (const void *)err}) fake::use(p, s);
  return cudaSuccess;
}
cudaError_t launch_advect_tiles(int, const TileArgs &a, int, TileShape, cudaStream_t s, bool) {
  if (!step_launch()) return cudaErrorInvalidValue;
  fake::use(a.out, s);
  return cudaSuccess;
}
cudaError_t launch_cell_words(const double *, const uint8_t *, double, long long, double *cell, cudaStream_t s) {
  fake::use(cell, s);
  return cudaSuccess;
}
cudaError_t launch_repitch(const void *, int, long long, long long, void *, int, long long, long long, int, int, int,
                           cudaStream_t) {
  return cudaSuccess;
}
cudaError_t launch_content(const void *, int, const void *, const void *, int, const double *, const double *,
                           const double *, const uint8_t *, int, int, int, int, long long, int, int, double, double *,
                           cudaStream_t) {
  return cudaSuccess;
}
cudaError_t launch_diff_table(const double *, const double *, const double *, const double *, const uint8_t *, double,
                              int, int, int, float2 *, cudaStream_t) {
  return cudaSuccess;
}
cudaError_t launch_wait_probe(int, int *, cudaStream_t) { return cudaSuccess; }

}  // namespace hyc
