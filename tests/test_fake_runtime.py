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
// fake_fail_after: allocations that still succeed (-1: all)
int fake_fail_after = -1, fake_mallocs, fake_frees, fake_graphs;
int cudaMalloc(void **p, size_t n) {
  if (fake_fail_after == 0) return 2;
  if (fake_fail_after > 0) fake_fail_after--;
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
int cudaStreamGetCaptureInfo_v2(void *s, int *st, unsigned long long *id, void **g, void **deps,
                                size_t *n) {
  *st = 1;
  if (g) *g = (void *)1;
  if (deps) *deps = NULL;
  if (n) *n = 0;
  return 0;
}
int cudaStreamEndCapture(void *s, void **g) { *g = (void *)1; return 0; }
// (type, reserved, then of a conditional node: handle, type, size, bodies out)
struct node { int type, reserved[3]; unsigned long long handle; int kind; unsigned size; void **out; };
int cudaGraphAddNode(void **n, void *g, void *d, size_t nd, struct node *p) {
  static void *body = (void *)1;
  p->out = &body;
  *n = (void *)1;
  return 0;
}
int cudaGraphInstantiate(void **e, void *g, unsigned long long f) {
  fake_graphs++;
  *e = (void *)1;
  return 0;
}
int cudaGraphExecDestroy(void *e) { fake_graphs--; return 0; }
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


def _count(fake, name):
    return C.c_int.in_dll(fake, name).value


def _fail_after(fake, n):
    C.c_int.in_dll(fake, "fake_fail_after").value = n


@pytest.fixture
def handle(fake, monkeypatch):
    """Makes a handle of a grid that is all tail."""
    monkeypatch.setattr(L, "_lib", fake)

    def make(precision):
        return RichardsGPU(configs.box(nx=12, ny=10, nz=8, nsteps=1), precision=precision)

    yield make
    _fail_after(fake, -1)


@pytest.mark.parametrize("precision, change", [("fp64", "max_iter"), ("mixed", "max_iter"),
                                               ("mixed16", "max_iter"), ("fp64", "full_jacobian")])
def test_level_leaves_the_tail_without_memory(fake, handle, precision, change):
    """A grid that is all tail: MGSemi.MaxIter 2 and FullJacobian take level 0
    out of the single-block kernel.  The V-cycle graph of the moment points to
    that kernel's packed operators, so they must not be freed before it goes;
    a change that cannot allocate leaves them alone."""
    g = handle(precision)
    frees = _count(fake, "fake_frees")
    _fail_after(fake, 0)
    if change == "max_iter":
        assert fake.pfgpu_set_mg_max_iter(g.h, 2) == 0
        assert fake.pfgpu_set_mg_max_iter(g.h, 1) == 0
    else:  # its own arrays are missing: refused, nothing changed
        assert fake.pfgpu_set_pc_matrix(g.h, 1) < 0
    assert _count(fake, "fake_frees") == frees
    _fail_after(fake, -1)
    g.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_full_jacobian_allocates_all_or_nothing(fake, handle, precision):
    """FullJacobian's arrays, with the allocator failing at each of them in
    turn: the call is refused, a later one completes the set, and none leaks."""
    live = lambda: _count(fake, "fake_mallocs") - _count(fake, "fake_frees")
    before = live()
    g = handle(precision)
    assert fake.pfgpu_set_pc_matrix(g.h, 1) == 0
    full = live() - before
    needed = 3 + 2 * len(g.mg_levels())
    g.close()
    assert live() == before
    for n in range(needed):
        g = handle(precision)
        _fail_after(fake, n)
        assert fake.pfgpu_set_pc_matrix(g.h, 1) < 0
        _fail_after(fake, -1)
        assert fake.pfgpu_set_pc_matrix(g.h, 1) == 0
        assert live() - before == full, n
        g.close()
        assert live() == before


def test_captured_solves_go_with_the_arrays_they_hold(fake, handle):
    """Back from FullJacobian the W, S and L of level 0 are freed: a solve
    captured with them must not be kept for its return."""
    base = _count(fake, "fake_graphs")
    g = handle("fp64")
    one = _count(fake, "fake_graphs") - base  # the V-cycle
    stats = L.Stats()
    for _ in range(2):
        assert fake.pfgpu_set_pc_matrix(g.h, 1) == 0
        fake.pfgpu_advance(g.h, C.c_double(0.1), 1, C.byref(stats))
        assert _count(fake, "fake_graphs") - base == one + 1  # and the solve
        assert fake.pfgpu_set_pc_matrix(g.h, 0) == 0
        assert _count(fake, "fake_graphs") - base == one
    g.close()
    assert _count(fake, "fake_graphs") == base
