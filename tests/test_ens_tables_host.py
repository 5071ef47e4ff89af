"""The FP64 ensemble's host layer (csrc/hyc_ens_host.cpp) against a CUDA
runtime in host memory (tests/host/fake_cuda.h): tensor maps are encoded, and
tile shapes are timed, only where a launch goes to a tile kernel."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "hycom-src_gb300", "csrc")
HOST = os.path.join(ROOT, "tests", "host")

SRC = r"""
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "hycom_adv.h"
#include "fake_cuda.h"
#include "fake_launch.h"
#define OK(x) do { if ((x) != HYC_OK) { printf("%s failed: %s\n", #x, hyc_ens_last_error(e)); return 2; } } while (0)
int main(int, char **argv) {
  const int advtyp = atoi(argv[1]), nx = 40, ny = 30, nb = 6, n = (nx + 2 * nb) * (ny + 2 * nb);
  fake_strip = atoi(argv[2]);
  std::vector<int> land(n, 0);
  std::vector<double> one(n, 1.0);
  hyc_basin_spec s = {nx, ny, 2, nb, 0, 3, land.data(), land.data(), land.data(), one.data(), one.data()};
  hyc_ens *e = nullptr;
  OK(hyc_ens_create(&e, 1, &s, HYC_PREC_FP64, 0));
  OK(hyc_ens_set_tile(e, 16, 16));
  OK(hyc_ens_step(e, 2, 1800.0, 1, 0));  // the queue needs none
  const int m0 = fake_maps;
  OK(hyc_ens_step(e, advtyp, 1800.0, 1, 0));
  OK(hyc_ens_step(e, advtyp, 1800.0, 2, 1));
  OK(hyc_ens_step(e, 2, 900.0, 1, 0));
  OK(hyc_ens_step(e, advtyp, 1800.0, 1, 0));
  const int m1 = fake_maps;
  int tx, ty;
  double ms;
  fake_step_launches = 0;
  OK(hyc_ens_tune(e, advtyp, 1800.0, &tx, &ty, &ms));
  printf("%d %d %d", m0, m1, fake_step_launches);
  if (fake_step_launches == 4) printf(" %dx%d", tx, ty);
  printf("\n");
  hyc_ens_destroy(e);
  return fake::dead_uses() || fake::bytes_in_use();
}
"""


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    d = tmp_path_factory.mktemp("ens_tables")
    (d / "t.cpp").write_text(SRC)
    out = str(d / "t")
    subprocess.run(["g++", "-O1", "-std=c++17", "-o", out, str(d / "t.cpp"), os.path.join(CSRC, "hyc_ens_host.cpp"),
                    os.path.join(HOST, "fake_cuda.cpp"), os.path.join(HOST, "fake_launch.cpp"), "-I", HOST, "-I", CSRC,
                    "-I", os.path.join(ROOT, "include"), "-I", "/usr/local/cuda/include"], check=True)
    return out


# three tracers: 3 rotations x (5 maps of the layer's arrays + 2 a tracer); the tuner's warm-up and 3 runs a shape
MAPS = 3 * (5 + 2 * 3)


@pytest.mark.parametrize("advtyp,strip,want", [(2, 1, "0 0 4 16x16"), (4, 1, "0 0 4 16x16"), (0, 1, "0 0 4 16x16"),
                                               (1, 1, "0 0 4 16x16"), (1, 0, f"0 {2 * MAPS} 8")])
def test_maps_and_shapes(exe, advtyp, strip, want):
    r = subprocess.run([exe, str(advtyp), str(strip)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == want, f"{r.returncode}: {r.stdout}"
