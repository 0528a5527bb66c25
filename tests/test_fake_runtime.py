"""Host paths of the library whose CUDA calls fail, on the CPU: the library's
objects linked against a stand-in for the CUDA runtime whose device memory is
host memory, whose kernels do nothing and whose allocator can be told to fail."""

import ctypes as C
import glob
import os
import subprocess

import pytest

from parflow_b200 import build as pbuild
from parflow_b200 import configs
from parflow_b200 import lib as L
from parflow_b200.solver import RichardsGPU

RUNTIME = r"""
#include <stdlib.h>
#include <string.h>
#include <stddef.h>
int fake_fail_malloc, fake_mallocs, fake_frees;
int cudaMalloc(void **p, size_t n) {
  if (fake_fail_malloc) return 2;
  fake_mallocs++;
  return (*p = calloc(1, n)) ? 0 : 2;
}
int cudaFree(void *p) { if (p) fake_frees++; free(p); return 0; }
int cudaMallocHost(void **p, size_t n) { return (*p = calloc(1, n)) ? 0 : 2; }
int cudaHostAlloc(void **p, size_t n, unsigned f) { return (*p = calloc(1, n)) ? 0 : 2; }
int cudaFreeHost(void *p) { free(p); return 0; }
int cudaMemcpy(void *d, const void *s, size_t n, int k) { memcpy(d, s, n); return 0; }
int cudaMemcpyAsync(void *d, const void *s, size_t n, int k, void *st) { memcpy(d, s, n); return 0; }
int cudaMemset(void *d, int v, size_t n) { memset(d, v, n); return 0; }
int cudaMemsetAsync(void *d, int v, size_t n, void *st) { memset(d, v, n); return 0; }
int cudaDeviceGetAttribute(int *v, int a, int d) { *v = 1; return 0; }
int cudaGetDevice(int *d) { *d = 0; return 0; }
int cudaPointerGetAttributes(void *a, const void *p) { return 1; }
const char *cudaGetErrorString(int e) { return "fake"; }
int cudaStreamCreateWithFlags(void **s, unsigned f) { *s = (void *)1; return 0; }
int cudaStreamEndCapture(void *s, void **g) { *g = (void *)1; return 0; }
int cudaGraphInstantiate(void **e, void *g, unsigned long long f) { *e = (void *)1; return 0; }
int cudaEventCreate(void **e) { *e = (void *)1; return 0; }
int cudaOccupancyMaxPotentialClusterSize(int *n, const void *f, const void *c) { *n = 1; return 0; }
int cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *f, int t, size_t s,
                                                           unsigned fl) { *n = 1; return 0; }
void **__cudaRegisterFatBinary(void *p) { static void *h; return &h; }
int __cudaPushCallConfiguration() { return 1; }
int __cudaPopCallConfiguration() { return 1; }
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    d = tmp_path_factory.mktemp("fake_runtime")
    objs = sorted(glob.glob(os.path.join(pbuild.HERE, "_build", "*.cu.o")))
    if len(objs) != len(pbuild.sources()) or not pbuild.up_to_date():
        pbuild.build(force=True)
        objs = sorted(glob.glob(os.path.join(pbuild.HERE, "_build", "*.cu.o")))
    text = RUNTIME
    wanted = set()
    for line in subprocess.check_output(["nm", "-u"] + objs, text=True).splitlines():
        name = line.split()[-1] if line.split() else ""
        if name.startswith(("cuda", "__cuda")):
            wanted.add(name)
    for name in sorted(wanted):  # everything else succeeds and does nothing
        if name + "(" not in RUNTIME:
            text += "int %s() { return 0; }\n" % name
    src, obj, so = (str(d / n) for n in ("rt.c", "rt.o", "libpfgpu_fake.so"))
    with open(src, "w") as f:
        f.write(text)
    subprocess.check_call(["gcc", "-w", "-fPIC", "-c", src, "-o", obj])
    subprocess.check_call([pbuild.nvcc()] + pbuild.ARCH + ["-shared", "-cudart", "none", "-o", so,
                                                           "-Xlinker", "-Bsymbolic", obj] + objs)
    kept, L._lib = L._lib, None
    lib = L.load(so)
    L._lib = kept
    return lib


@pytest.mark.parametrize("precision, change", [("fp64", "max_iter"), ("mixed", "max_iter"),
                                               ("mixed16", "max_iter"), ("fp64", "full_jacobian")])
def test_level_leaves_the_tail_without_memory(fake, monkeypatch, precision, change):
    """A grid that is all tail: MGSemi.MaxIter 2 and FullJacobian take level 0
    out of the single-block kernel.  The V-cycle graph of the moment points to
    that kernel's packed operators, so they must not be freed before it goes;
    a change that cannot allocate leaves them alone."""
    monkeypatch.setattr(L, "_lib", fake)
    g = RichardsGPU(configs.box(nx=12, ny=10, nz=8, nsteps=1), precision=precision)
    count = lambda name: C.c_int.in_dll(fake, name).value
    frees = count("fake_frees")
    C.c_int.in_dll(fake, "fake_fail_malloc").value = 1
    try:
        if change == "max_iter":
            assert fake.pfgpu_set_mg_max_iter(g.h, 2) == 0
            assert fake.pfgpu_set_mg_max_iter(g.h, 1) == 0
        else:  # its own arrays are missing: refused, nothing changed
            assert fake.pfgpu_set_pc_matrix(g.h, 1) < 0
        assert count("fake_frees") == frees
    finally:
        C.c_int.in_dll(fake, "fake_fail_malloc").value = 0
        g.close()
