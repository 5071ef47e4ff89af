"""cnuity's layers per launch: as many as 1 GiB of work slices holds, at least
one, and no more than a launch's grid takes."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LIBDIR = os.path.join(ROOT, "hycom-src_gb300", "hycadv", "_lib")


def test_batch_limits(built_lib, tmp_path):
    exe = str(tmp_path / "batch")
    subprocess.run(["g++", "-O1", "-std=c++17", "-o", exe, os.path.join(ROOT, "tests", "host", "batch.cpp"),
                    "-I", os.path.join(ROOT, "hycom-src_gb300", "csrc"), "-I", "/usr/local/cuda/include",
                    os.path.join(LIBDIR, "libhycadv.so"), f"-Wl,-rpath,{LIBDIR}", "-Wl,--unresolved-symbols=ignore-all"],
                   check=True)
    cases = [(169, 41, 41), (169, 100000, 65535), (712 * 612, 45, 44), (4512 * 3310, 41, 1), (4 * 10 ** 9, 3, 1)]
    args = [str(v) for cells, layers, _ in cases for v in (cells, layers)]
    out = subprocess.run([exe] + args, capture_output=True, text=True, timeout=60, check=True).stdout.split()
    assert [int(v) for v in out] == [want for *_, want in cases]
