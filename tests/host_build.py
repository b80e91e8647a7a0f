"""Builds a C file of the host layer with fakes in place of the CUDA runtime and
the kernel launchers (tests/host_fakes.c), for tests that need no GPU."""
import ctypes as C
import os
import subprocess

from n_body_sim_pro_b200 import build as B

TESTS = os.path.dirname(os.path.abspath(__file__))


def build(folder, unit, fakes):
    """A loaded library of csrc/`unit` and the C text `fakes`; every function that is
    still undefined returns 0."""
    src = os.path.join(folder, "unit.c")
    with open(src, "w") as f:
        f.write(f'#include "{unit}"\n#include "host_fakes.c"\n#define EXPORT __attribute__((visibility("default")))\n{fakes}\n')
    obj, stubs, lib = (os.path.join(folder, name) for name in ("unit.o", "stubs.c", "libunit.so"))
    cc = [B._cc(), "-std=gnu17", "-O1", "-fPIC", "-fvisibility=hidden"]
    subprocess.run(cc + ["-I" + B.CSRC, "-I" + B.INCLUDE, "-I" + TESTS,
                         "-I" + os.path.join(B._cuda_home(), "include"), "-c", src, "-o", obj], check=True)
    missing = subprocess.run(["nm", "-u", obj], check=True, capture_output=True, text=True).stdout.split()
    missing = [s for s in missing if s.startswith(("cuda", "nbsp_", "n_body_"))]
    with open(stubs, "w") as f:
        f.writelines(f"long {s}(void) {{ return 0; }}\n" for s in missing)
    subprocess.run(cc + ["-shared", "-Wl,-Bsymbolic", "-o", lib, obj, stubs, "-lm"], check=True)
    return C.CDLL(lib)
