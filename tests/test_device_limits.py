"""What the library asks of the CUDA runtime, which is replaced by a stand-in of
two devices that records it; no GPU is touched.

Launch limits: function attributes belong to a device, so a context has to set on
its own device what another has set on another one.  Copies: those of the particle
state hold what crosses the interface."""
from __future__ import annotations

import re
import subprocess
import sys
from pathlib import Path

import pytest

from interparts_mpich_gb300 import build as b

ROOT = Path(__file__).resolve().parents[1]

SPECIAL = r"""
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
int fake_device = 0;
int cudaGetDevice(int *d) { *d = fake_device; return 0; }
int cudaFuncSetAttribute(const void *f, int attr, int value) {
  printf("%d %p %d %d\n", fake_device, f, attr, value);
  fflush(stdout);
  return 0;
}
int cudaMalloc(void **p, size_t n) { *p = calloc(n, 1); return 0; }
int cudaMallocHost(void **p, size_t n) { *p = calloc(n, 1); return 0; }
int cudaFree(void *p) { free(p); return 0; }
int cudaFreeHost(void *p) { free(p); return 0; }
int cudaMemcpyAsync(void *d, const void *s, size_t n, int k, void *st) {
  printf("copy %zu\n", n);
  fflush(stdout);
  memcpy(d, s, n);
  return 0;
}
int cudaStreamCreateWithFlags(void **s, unsigned f) { *s = &fake_device; return 0; }
int cudaEventCreate(void **e) { *e = &fake_device; return 0; }
int cudaDeviceGetAttribute(int *v, int a, int d) { *v = 152; return 0; }
const char *cudaGetErrorString(int e) { return ""; }
void **__cudaRegisterFatBinary(void *f) { static void *h; return &h; }
"""

START = """
import ctypes, sys
rt = ctypes.CDLL(sys.argv[1])
from interparts_mpich_gb300 import IBM_MODE_MIXED_LEARNED, IBMSolver
from interparts_mpich_gb300.cases import Case
"""
LIMITS = START + """
for d in (0, 1):
    ctypes.c_int.in_dll(rt, "fake_device").value = d
    IBMSolver(Case(name="limits", itot=64, jtot=64, ktot=64, radius=11.0 / 64, np=2, visc=1e-2),
              mode=IBM_MODE_MIXED_LEARNED).close()
"""
COPIES = START + """
case = Case(name="copies", itot=64, jtot=64, ktot=64, radius=2.0 / 64, np=97, visc=1e-2)
s = IBMSolver(case)
ps = case.initial_particles(lagrangian=False)
print("begin", flush=True)
s.set_particles(ps)
s.get_particles(lagrangian=False)
print("end", flush=True)
"""


def run_on_fake_runtime(program, tmp_path) -> list[str]:
    lib = b.build()
    nm = subprocess.run(["nm", "-D", "--undefined-only", str(lib)], check=True, capture_output=True, text=True).stdout
    names = set(re.findall(r" U (_*cuda\w+)", nm))
    if not names:
        pytest.skip("the CUDA runtime is linked in")
    rest = "".join(f"int {n}() {{ return 0; }}\n" for n in sorted(names) if not re.search(rf"\b{n}\(", SPECIAL))
    src, fake, ver = tmp_path / "fake.c", tmp_path / "libcudart.so.13", tmp_path / "map"
    src.write_text(SPECIAL + rest)
    ver.write_text("libcudart.so.13 { *; };\n")
    subprocess.run(["gcc", "-shared", "-fPIC", "-w", str(src), "-o", str(fake), "-Wl,-soname,libcudart.so.13",
                    f"-Wl,--version-script={ver}"], check=True)
    r = subprocess.run([sys.executable, "-c", program, str(fake)], cwd=ROOT, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr
    return r.stdout.splitlines()


def test_limits_are_set_on_each_device(tmp_path):
    sets = [line.split(" ", 1) for line in run_on_fake_runtime(LIMITS, tmp_path)]
    a, c = ({s for d, s in sets if d == q} for q in "01")
    assert len(a) > 20 and a == c


def test_particle_copies(tmp_path):
    """The 31 fields of a particle and the 24 of its last substep go in and come
    out, the collision pass's snapshots do not."""
    lines = run_on_fake_runtime(COPIES, tmp_path)
    lines = lines[lines.index("begin"):lines.index("end")]
    sizes = [int(line.split()[1]) for line in lines if line.startswith("copy")]
    assert sizes.count(55 * 97 * 8) == 2 and not any(55 * 97 * 8 < n <= 80 * 97 * 8 for n in sizes), sizes
