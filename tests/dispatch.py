"""The kernel that a launch of the plain FP64 form goes to (tests/host/dispatch.cpp)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LIBDIR = os.path.join(ROOT, "hycom-src_gb300", "hycadv", "_lib")


def build(d):
    """The compiled question, in directory d; libhycadv.so has to be built."""
    out = os.path.join(str(d), "dispatch")
    subprocess.run(["g++", "-O1", "-std=c++17", "-o", out, os.path.join(ROOT, "tests", "host", "dispatch.cpp"),
                    "-I", os.path.join(ROOT, "hycom-src_gb300", "csrc"), "-I", "/usr/local/cuda/include",
                    os.path.join(LIBDIR, "libhycadv.so"), f"-Wl,-rpath,{LIBDIR}", "-Wl,--unresolved-symbols=ignore-all"],
                   check=True)
    return out


def routes(exe, launches, shape="free"):
    """launches: (scheme, ii, jj, layers, fields) each; a route each."""
    args = [str(v) for x in launches for v in x]
    r = subprocess.run([exe, shape] + args, capture_output=True, text=True, timeout=120, check=True)
    return r.stdout.splitlines()
