"""cnuity's work slices on a device that is nearly full: the host layer
(csrc/hyc_host.cpp) against a CUDA runtime in host memory
(tests/host/fake_cuda.h)."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "hycom-src_gb300", "csrc")
HOST = os.path.join(ROOT, "tests", "host")

SRC = r"""
#include <cuda_runtime.h>
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "hycom_adv.h"
#include "hyc_args.h"
#include "hyc_internal.h"
#include "fake_cuda.h"
static int batch = -1;
static bool inside = true;
namespace hyc {  // the kernels' side: 9 slices, and 7 for each layer of a batch
int mass_sum_partials() { return 8; }
double key_to_double(long long) { return 0.0; }
long long double_to_key(double) { return 0; }
bool advect_tile_shape_ok(TileShape) { return true; }
int cnuity_batch(long long, int kdm) { return kdm; }
size_t cnuity_work_slices(int n) { return 9 + 7 * (size_t)n; }
cudaError_t launch_xctilr_list(const std::vector<std::pair<double *, int>> &, long long, int, int, int, int, int, int, int,
                               int *, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_cnuity_layers(const CnuityArgs &a, int *, cudaStream_t s) {
  batch = a.nbatch;
  fake::use(a.w, s);
  fake::use(a.w + cnuity_work_slices(batch) * a.slice - 1, s);
  return cudaGetLastError();  // as the launchers end
}
cudaError_t launch_cnuity_rest(const CnuityArgs &, int *, cudaStream_t) { return cudaGetLastError(); }
}
#define OK(x) do { if ((x) != HYC_OK) { printf("%s failed\n", #x); return 2; } } while (0)
int main(int, char **argv) {
  const int nx = 20, ny = 18, nb = 6, kdm = 12, ld = nx + 2 * nb, n = ld * (ny + 2 * nb);
  std::vector<int> land(n, 0);
  std::vector<double> one(n, 1.0);
  hyc_ctx *c = nullptr;
  OK(hyc_adv_init(&c, nx, ny, kdm, nb, 0, land.data(), land.data(), land.data(), one.data(), one.data(), 0));
  OK(hyc_set_cnuity_grid(c, one.data(), one.data(), one.data(), one.data(), nullptr, nullptr));
  for (int f = 0; f < HYC_NFIELDS; f++) {
    void *p;
    cudaMalloc(&p, 8);
    OK(hyc_bind_field(c, f, p, (long long)n * 1000, HYC_DEVICE));
  }
  // free memory in slices
  fake::set_free_bytes((size_t)atoi(argv[1]) * n * 8);
  fake::hide_free(argv[2][0] == 'h');
  hyc_cnuity_params p = {1, 0, 0, 0, 600.0, 0.1};
  const size_t before = fake::bytes_in_use();
  const int rc = hyc_cnuity(c, 1, 2, &p, nullptr);
  printf("rc %d batch %d slices %zu dead %d\n", rc, batch, (fake::bytes_in_use() - before) / (n * 8), fake::dead_uses());
  if (rc == HYC_OK) OK(hyc_cnuity(c, 2, 1, &p, nullptr));
  return 0;
}
"""


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    d = tmp_path_factory.mktemp("cnuity_host")
    (d / "t.cpp").write_text(SRC)
    out = str(d / "t")
    subprocess.run(["g++", "-O1", "-std=c++17", "-o", out, str(d / "t.cpp"), os.path.join(CSRC, "hyc_host.cpp"),
                    os.path.join(HOST, "fake_cuda.cpp"), "-I", HOST, "-I", CSRC, "-I", os.path.join(ROOT, "include"),
                    "-I", "/usr/local/cuda/include", "-Wl,--unresolved-symbols=ignore-all"], check=True)
    return out


@pytest.mark.parametrize("free,shown,batch", [
    (10 ** 6, "shown", 12),  # plenty
    (16 * 93, "shown", 12),  # a sixteenth holds 9 + 7*12 slices
    (16 * 60, "shown", 7),   # 9 + 7*7 = 58
    (200, "shown", 1),       # even one layer's 16 slices are more than a sixteenth
    (40, "hidden", 3),       # the free memory is not what can be had: 12, 6, then 3 layers
    (16, "hidden", 1),
    (15, "hidden", 0),       # not one layer: an error
])
def test_batch_follows_the_memory(exe, free, shown, batch):
    r = subprocess.run([exe, str(free), shown], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
    want = f"rc 0 batch {batch} slices {9 + 7 * batch} dead 0" if batch else "rc -9 batch -1 slices 0 dead 0"
    assert r.stdout.splitlines()[0] == want
