"""The ensemble's host layer (csrc/hyc_ens_host.cpp) against a CUDA runtime in
host memory (tests/host/fake_cuda.h): a step graph is not replayed once a
buffer that it was recorded with has been replaced."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "hycom-src_gb300", "csrc")
HOST = os.path.join(ROOT, "tests", "host")

SRC = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>
#include "hycom_adv.h"
#include "fake_cuda.h"
#include "fake_launch.h"
#define OK(x) do { if ((x) != HYC_OK) { printf("%s failed: %s\n", #x, hyc_ens_last_error(e)); return 2; } } while (0)
int main(int, char **argv) {
  const int prec = atoi(argv[2]), nx = 40, ny = 30, nb = 6, n = (nx + 2 * nb) * (ny + 2 * nb), ld = nx + 2 * nb;
  std::vector<int> ip(n, 0), iu(n, 0), iv(n, 0);
  std::vector<double> one(n, 1.0);
  for (int j = nb + 1; j < nb + ny - 1; j++)
    for (int i = nb + 1; i < nb + nx - 1; i++) ip[i + j * ld] = 1;
  for (int t = ld; t < n; t++) iu[t] = ip[t] && ip[t - 1], iv[t] = ip[t] && ip[t - ld];
  hyc_basin_spec s = {nx, ny, 2, nb, 0, 3, ip.data(), iu.data(), iv.data(), one.data(), one.data()};
  hyc_ens *e = nullptr;
  OK(hyc_ens_create(&e, 1, &s, prec, 0));
  if (!strcmp(argv[1], "longer-run")) {  // more queue counters than the graph was recorded with
    OK(hyc_ens_step(e, 2, 1800.0, 3, 1));
    OK(hyc_ens_step(e, 2, 1800.0, 5, 0));
    OK(hyc_ens_step(e, 2, 1800.0, 1, 0));  // back to the rotation of the graph
    OK(hyc_ens_step(e, 2, 1800.0, 3, 1));
  } else if (!strcmp(argv[1], "failed-tune")) {  // the tuner replaces the queue, then fails
    OK(hyc_ens_step(e, 2, 1800.0, 3, 1));
    int tx, ty;
    double ms;
    fake_strip = false;      // MPDATA in the tile kernel: two shapes
    fake_fail_launches = 6;  // the second one's
    if (hyc_ens_tune(e, 1, 1800.0, &tx, &ty, &ms) == HYC_OK) return 3;
    OK(hyc_ens_step(e, 2, 1800.0, 3, 1));
  } else if (!strcmp(argv[1], "no-memory")) {  // the queue counters cannot grow
    OK(hyc_ens_step(e, 2, 1800.0, 3, 1));
    fake::set_free_bytes(0);
    if (hyc_ens_step(e, 2, 1800.0, 1000, 0) == HYC_OK) return 4;
    fake::set_free_bytes(1 << 30);
    OK(hyc_ens_step(e, 2, 1800.0, 3, 1));
    OK(hyc_ens_step(e, 2, 1800.0, 3, 0));
  } else {  // nothing replaced: one graph serves both runs
    OK(hyc_ens_step(e, 2, 1800.0, 3, 1));
    OK(hyc_ens_step(e, 2, 1800.0, 3, 1));
    if (fake::captures() != 1) return 5;
  }
  printf("%d uses of freed memory, %d captures\n", fake::dead_uses(), fake::captures());
  hyc_ens_destroy(e);
  return fake::dead_uses() || fake::graph_launches() != 2 || fake::bytes_in_use();
}
"""


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    d = tmp_path_factory.mktemp("ens_host")
    (d / "t.cpp").write_text(SRC)
    out = str(d / "t")
    subprocess.run(["g++", "-O1", "-std=c++17", "-o", out, str(d / "t.cpp"), os.path.join(CSRC, "hyc_ens_host.cpp"),
                    os.path.join(HOST, "fake_cuda.cpp"), os.path.join(HOST, "fake_launch.cpp"), "-I", HOST, "-I", CSRC,
                    "-I", os.path.join(ROOT, "include"), "-I", "/usr/local/cuda/include"], check=True)
    return out


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("how", ["reuse", "longer-run", "failed-tune", "no-memory"])
def test_graph_and_its_buffers(exe, how, precision):
    r = subprocess.run([exe, how, str(precision)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, f"{r.returncode}: {r.stdout}"
