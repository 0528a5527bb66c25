"""ModifiedGS's second pass (a new Krylov vector that the projections cancelled,
as at an exact breakdown): over the whole grid for long vectors, in the cluster
for short ones, and in a solve that meets it (an impermeable domain, whose
Jacobian is diagonal, so that M^-1 is its inverse)."""

import ctypes as C
import math
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
FINISH = "_ZN5pfgpu19launch_gmres_finishEPKPdiixS0_S0_PiP11CUstream_stPNS_7NkStateEPKNS_7NkCondsE"
MGS = "_ZN5pfgpu16launch_gmres_mgsEPKPdiixS0_P11CUstream_stPNS_7NkStateEPKNS_7NkCondsE"
LMAX = 12
RNORM, ROT, RHO, VKNORM2, NEWNORM2, HLL = range(6)
EPS = 2.0 ** -53


@pytest.fixture(scope="module")
def torch():
    t = pytest.importorskip("torch")
    if not t.cuda.is_available():
        pytest.fail("CUDA device required for gpu tests")
    from parflow_b200 import configs
    from parflow_b200.solver import RichardsGPU

    RichardsGPU(configs.box(nx=4, ny=4, nz=4, nsteps=1)).close()  # (prepares the kernels)
    return t


class Scalars:
    """The scalar block of GMRES on the device (Hessenberg matrix, rotations,
    right-hand side, named scalars) with room for the second pass's words."""

    def __init__(self, torch, l, h, rng):
        self.nh, self.ngiv = (LMAX + 1) * LMAX, (LMAX + 1) * LMAX + 2 * LMAX
        self.sc = self.ngiv + LMAX + 1
        s = np.zeros(self.sc + 512)
        s[:self.nh].reshape(LMAX + 1, LMAX)[:l + 1, l] = h
        ang = rng.uniform(0.0, 2.0 * math.pi, l)
        s[self.nh:self.nh + 2 * l:2], s[self.nh + 1:self.nh + 2 * l:2] = np.cos(ang), np.sin(ang)
        s[self.sc + RNORM], s[self.sc + ROT] = 3.0, 0.5
        self.start = s
        self.dev = torch.tensor(s, device="cuda")

    def reset(self, torch, vk2=0.0, new2=0.0):
        s = self.start.copy()
        s[self.sc + VKNORM2], s[self.sc + NEWNORM2] = vk2, new2
        self.dev[:self.sc + 8] = torch.tensor(s[:self.sc + 8], device="cuda")

    def read(self):
        return self.dev.cpu().numpy()


def _column(s, start, l, h, hk):
    """Column l after the earlier rotations and its own (iterativ.c:205-250)."""
    h = list(h) + [hk]
    for i in range(l):
        c, sn = start[s.nh + 2 * i], start[s.nh + 2 * i + 1]
        h[i], h[i + 1] = c * h[i] - sn * h[i + 1], sn * h[i] + c * h[i + 1]
    t1, t2 = h[l], h[l + 1]
    if abs(t2) >= abs(t1):
        sn = -1.0 / math.sqrt(1.0 + (t1 / t2) ** 2)
        c = -sn * (t1 / t2)
    else:
        c = 1.0 / math.sqrt(1.0 + (t2 / t1) ** 2)
        sn = -c * (t2 / t1)
    h[l], h[l + 1] = c * t1 - sn * t2, t2
    return h, abs(0.5 * sn * 3.0)


def _basis(torch, n, k, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    q = torch.linalg.qr(torch.randn(n, k + 1, generator=g, device="cuda", dtype=torch.float64))[0]
    return [q[:, i].contiguous() for i in range(k + 1)]  # the last: outside the basis


def _pointers(vs):
    return (C.c_void_p * len(vs))(*[v.data_ptr() for v in vs])


@pytest.mark.parametrize("n, l", [(1000, 2), (65537, 0), (70001, 3), (606208, 1), (606209, 9)])
def test_long_vector(torch, n, l):
    """Every product is taken off, in order, but the one below rounding of its
    coefficient; the same bits on a second launch (its words were cleared)."""
    from parflow_b200 import lib as L

    fn = getattr(L.load(), FINISH)
    fn.restype = None
    k = l + 1
    rng = np.random.default_rng(n + l)
    *basis, w = _basis(torch, n, k, n + l)
    a = rng.uniform(0.1, 0.5, k)
    h = rng.uniform(-1.0, 1.0, k)
    if k > 2:
        a[1], h[1] = 1e-13, 1e3  # too small beside its coefficient: stays in
    vk0 = w + sum(float(c) * v for c, v in zip(a, basis))
    # the second pass on the host
    want, want_h, nn2 = vk0.cpu().numpy().copy(), h.copy(), 0.0
    for i in range(k):
        v = basis[i].cpu().numpy()
        p = float(np.dot(v, want))
        if 1000.0 * want_h[i] + p != 1000.0 * want_h[i]:
            want_h[i] += p
            nn2 += p * p
            want -= p * v
    norm2 = float(torch.dot(vk0, vk0))
    hk = math.sqrt(norm2 - nn2)
    s = Scalars(torch, l, h, rng)
    partial = torch.zeros(4 * 592, device="cuda", dtype=torch.float64)
    err = torch.zeros(1, device="cuda", dtype=torch.int32)
    got = []
    for _ in range(2):
        vk = vk0.clone()
        vs = _pointers(basis + [vk])
        s.reset(torch, 1e32, norm2)
        torch.cuda.synchronize()
        fn(vs, C.c_int(l), C.c_int(LMAX), C.c_longlong(n), C.c_void_p(s.dev.data_ptr()),
           C.c_void_p(partial.data_ptr()), C.c_void_p(err.data_ptr()), None, None, None)
        torch.cuda.synchronize()
        got.append((vk.cpu().numpy(), s.read()))
    assert int(err) == 0
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])
    x, sc = got[0]
    assert not sc[s.sc + 8:].any()  # the words of the second pass
    # a product of n terms errs by n eps |v| |vk| at most (|vk| < 2), and the
    # errors of k of them meet in vk
    tol = 2.0 * n * EPS * k
    assert np.abs(x - want).max() <= tol
    col, rho = _column(s, s.start, l, want_h, hk)
    H = sc[:s.nh].reshape(LMAX + 1, LMAX)[:l + 2, l]
    # (the rotations: four roundings an entry, entries of up to 1e3)
    assert np.abs(H - col).max() <= 2 * tol + 8 * (l + 1) * EPS * 1e3
    assert abs(sc[s.sc + HLL] - hk) <= 4 * tol / hk
    # rho moves with the last rotation's angle: the errors of t1 and t2 over their length
    assert abs(sc[s.sc + RHO] - rho) <= 1.5 * (6 * tol + 8 * (l + 1) * EPS * 1e3) / hk


def test_long_vector_takes_the_whole_gpu(torch):
    """Eight million cells against four vectors: some 1 GB, 0.2 ms at the memory
    rate.  One block alone would take about 10 ms."""
    from parflow_b200 import lib as L

    fn = getattr(L.load(), FINISH)
    fn.restype = None
    n, l = 8000000, 3
    rng = np.random.default_rng(5)
    vs = [torch.zeros(n, device="cuda", dtype=torch.float64) for _ in range(l + 2)]
    for i, v in enumerate(vs):
        v[i::l + 2] = 1.0 / math.sqrt(n / (l + 2))
    vk0 = vs[-1] + 0.25 * sum(vs[:-1])
    s = Scalars(torch, l, rng.uniform(-1.0, 1.0, l + 1), rng)
    err = torch.zeros(1, device="cuda", dtype=torch.int32)
    partial = torch.zeros(4 * 592, device="cuda", dtype=torch.float64)
    best = math.inf
    for _ in range(4):
        vk = vk0.clone()
        s.reset(torch, 1e32, 1.25)
        ptrs = _pointers(vs[:-1] + [vk])
        ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        torch.cuda.synchronize()
        ev[0].record(torch.cuda.default_stream())
        fn(ptrs, C.c_int(l), C.c_int(LMAX), C.c_longlong(n), C.c_void_p(s.dev.data_ptr()),
           C.c_void_p(partial.data_ptr()), C.c_void_p(err.data_ptr()), None, None, None)
        ev[1].record(torch.cuda.default_stream())
        torch.cuda.synchronize()
        best = min(best, ev[0].elapsed_time(ev[1]))
    assert int(err) == 0 and float((vk - vs[-1]).abs().max()) <= 1e-12
    assert best < 2.0


def test_wait_that_runs_out(torch):
    """The sums of the first product are never made (its chunks are marked as
    claimed): every block gives up after a second, the launch ends with its
    error word set and its own words cleared, and the norm is no number."""
    from parflow_b200 import lib as L

    fn = getattr(L.load(), FINISH)
    fn.restype = None
    n, l = 70001, 1
    rng = np.random.default_rng(4)
    vs = _basis(torch, n, l + 1, 4)
    s = Scalars(torch, l, rng.uniform(-1.0, 1.0, l + 1), rng)
    s.reset(torch, 1e32, 1.0)
    s.dev[s.sc + 8:s.sc + 9].view(torch.int32)[0] = 1000000
    err = torch.zeros(1, device="cuda", dtype=torch.int32)
    partial = torch.zeros(4 * 592, device="cuda", dtype=torch.float64)
    torch.cuda.synchronize()
    fn(_pointers(vs), C.c_int(l), C.c_int(LMAX), C.c_longlong(n), C.c_void_p(s.dev.data_ptr()),
       C.c_void_p(partial.data_ptr()), C.c_void_p(err.data_ptr()), None, None, None)
    torch.cuda.synchronize()
    sc = s.read()
    assert int(err) == 4 and math.isnan(sc[s.sc + HLL]) and not sc[s.sc + 8:].any()


def test_vector_that_is_not_cancelled(torch):
    from parflow_b200 import lib as L

    fn = getattr(L.load(), FINISH)
    fn.restype = None
    n, l = 70001, 2
    rng = np.random.default_rng(3)
    vs = _basis(torch, n, l + 1, 3)
    h = rng.uniform(-1.0, 1.0, l + 1)
    s = Scalars(torch, l, h, rng)
    s.reset(torch, 1.0, 0.25)
    err = torch.zeros(1, device="cuda", dtype=torch.int32)
    partial = torch.zeros(4 * 592, device="cuda", dtype=torch.float64)
    before = vs[-1].clone()
    torch.cuda.synchronize()
    fn(_pointers(vs), C.c_int(l), C.c_int(LMAX), C.c_longlong(n), C.c_void_p(s.dev.data_ptr()),
       C.c_void_p(partial.data_ptr()), C.c_void_p(err.data_ptr()), None, None, None)
    torch.cuda.synchronize()
    assert torch.equal(vs[-1], before) and int(err) == 0
    sc = s.read()
    col, rho = _column(s, s.start, l, h, 0.5)
    H = sc[:s.nh].reshape(LMAX + 1, LMAX)[:l + 2, l]
    assert np.abs(H - col).max() <= 1e-14 and abs(sc[s.sc + RHO] - rho) <= 1e-14


@pytest.mark.parametrize("n, l", [(3000, 1), (9001, 4), (65536, 4)])
def test_short_vector(torch, n, l):
    """One launch for the whole Gram-Schmidt step (2, 8 and 8 blocks) of a vector
    that lies in the basis up to 1e-14 of its norm.  The first pass leaves
    products of 1e-17; beside coefficients that are zero up to rounding the
    second one takes them off down to rounding of what is left."""
    from parflow_b200 import lib as L

    fn = getattr(L.load(), MGS)
    fn.restype = None
    k = l + 1
    rng = np.random.default_rng(n + l)
    *basis, w = _basis(torch, n, k, n + l)
    a = np.zeros(k)
    a[l] = 1.0
    vk = basis[l] + 1e-14 * w
    before = [math.fsum((v * vk).tolist()) for v in basis]
    s = Scalars(torch, l, np.zeros(k), rng)
    s.reset(torch)
    torch.cuda.synchronize()
    fn(_pointers(basis + [vk]), C.c_int(l), C.c_int(LMAX), C.c_longlong(n),
       C.c_void_p(s.dev.data_ptr()), None, None, None)
    torch.cuda.synchronize()
    assert max(abs(b) for b in before[:l]) > 1e-19  # (they were there)
    norm = float(torch.linalg.vector_norm(vk))
    assert 0.5e-14 < norm < 5e-14
    for v in basis[:l]:
        # n eps of the product's terms, and what the later vectors bring back:
        # products of 1e-15 between vectors whose coefficients are below 1e-15
        assert abs(math.fsum((v * vk).tolist())) <= n * EPS * norm + 1e-29
    sc = s.read()
    assert abs(sc[s.sc + HLL] - norm) <= 1e-6 * norm


CHILD = r"""
import sys
sys.path.insert(0, sys.argv[1])
import numpy as np
from parflow_b200 import configs
from parflow_b200.solver import RichardsGPU
from oracle.oracle import Oracle
nx, ny, nz = (int(a) for a in sys.argv[2:5])
prob = configs.box(nx=nx, ny=ny, nz=nz, nsteps=2)
prob.perm = np.zeros(prob.shape)
po, so = Oracle(prob).run(2)
for graph in (0, 1):
    g = RichardsGPU(prob)
    g.solve_graph(graph)
    ps, st = g.run(2)
    assert [s.nonlin_iters for s in st] == [s.nni for s in so]
    assert [s.lin_iters for s in st] == [s.nli for s in so] == [s.nni for s in so]
    assert np.abs(ps[-1] - po[-1]).max() <= 1e-9 * np.abs(po[-1]).max()
    g.close()
"""


@pytest.mark.parametrize("shape, cells", [((64, 48, 24), "65536"), ((64, 48, 20), "65536"),
                                          ((64, 48, 20), "0")])
def test_solve_that_breaks_down(torch, shape, cells):
    """Every GMRES stops after one iteration, as the oracle's does."""
    env = dict(os.environ, PFGPU_MGS_CELLS=cells)
    subprocess.run([sys.executable, "-c", CHILD, ROOT] + [str(a) for a in shape], env=env,
                   check=True, timeout=300)
