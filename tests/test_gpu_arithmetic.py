"""The reciprocals and quotients of the residual, the Jacobian and the van
Genuchten pass against CUDA's division: within one unit in the last place,
equal where an operand is out of the range they are made for."""

import ctypes as C
import os

import numpy as np
import pytest

from parflow_b200 import build as pbuild

pytestmark = pytest.mark.gpu

RCP, QUOTIENT, QUOTIENT32 = range(3)
N = 1 << 21


@pytest.fixture(scope="module")
def check():
    import torch

    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for gpu tests")
    path = pbuild.CHECK_LIB
    if not os.path.exists(path):
        pbuild.build_checks()
    lib = C.CDLL(path)

    def run(op, a, b):
        a, b = np.broadcast_arrays(np.asarray(a, float), np.asarray(b, float))
        dev = [torch.tensor(np.ascontiguousarray(v), device="cuda") for v in (a, b)]
        dev += [torch.zeros_like(dev[0]) for _ in range(2)]
        assert lib.arith_check(op, *(C.c_void_p(v.data_ptr()) for v in dev),
                               C.c_longlong(b.size)) == 0
        return dev[2].cpu().numpy(), dev[3].cpu().numpy()

    def far(fp32, b):
        dev = [torch.tensor(np.ascontiguousarray(b, dtype=float), device="cuda")]
        dev.append(torch.zeros_like(dev[0]))
        assert lib.arith_far(fp32, *(C.c_void_p(v.data_ptr()) for v in dev),
                             C.c_longlong(dev[0].numel())) == 0
        return dev[1].cpu().numpy() != 0

    run.far = far
    return run


def _random(rng, lo, hi, n=N):
    """Random signs and significands, exponents lo .. hi - 1."""
    return np.ldexp(rng.uniform(1.0, 2.0, n) * rng.choice([-1.0, 1.0], n),
                    rng.integers(lo, hi, n).astype(np.int32))


def _within(got, want, b, fp32):
    """One unit of want, and what half of the smallest subnormal in the
    numerator makes (a correction below the normal range is lost)."""
    if fp32:
        unit = np.spacing(np.abs(want).astype(np.float32)).astype(float)
        sub = 2.0 ** -150
    else:
        unit, sub = np.spacing(np.abs(want)), 2.0 ** -1075
    with np.errstate(all="ignore"):
        # (2^-1075 is not a double: the product is taken in two factors)
        lost = sub / np.abs(b) if fp32 else (2.0 ** -1000 / np.abs(b)) * 2.0 ** -75
        err = np.abs(got - want)
        ok = (err <= unit + 1.01 * lost) | (got == want) | (np.isnan(got) & np.isnan(want))
    assert ok.all(), (got[~ok][:4], want[~ok][:4], b[~ok][:4])


def test_reciprocal(check):
    rng = np.random.default_rng(1)
    for lo, hi in ((-4, 4), (-1000, -996), (498, 503), (-999, 501), (-1074, 1024)):
        b = _random(rng, lo, hi)
        got, want = check(RCP, 0.0, b)
        _within(got, want, np.inf, False)
        far = check.far(0, b)
        assert np.array_equal(got[far], want[far])


def test_quotient(check):
    rng = np.random.default_rng(2)
    for b_range in ((-4, 4), (-1000, -996), (498, 503), (-999, 501)):
        for a_range in ((-4, 4), (-1074, -960), (-1022, 500)):
            a, b = _random(rng, *a_range), _random(rng, *b_range)
            got, want = check(QUOTIENT, a, b)
            use = np.isfinite(want)
            _within(got[use], want[use], b[use], False)
            far = check.far(0, b)
            assert np.array_equal(got[far], want[far])


def test_quotient_fp32(check):
    rng = np.random.default_rng(3)
    for b_range in ((-4, 4), (-113, -109), (60, 66), (-111, 63)):
        for a_range in ((-4, 4), (-149, -100), (-126, 60)):
            a, b = (_random(rng, *r).astype(np.float32).astype(float) for r in (a_range, b_range))
            got, want = check(QUOTIENT32, a, b)
            use = np.isfinite(want)
            _within(got[use], want[use], b[use], True)
            far = check.far(1, b)
            assert np.array_equal(got[far], want[far])


def test_range(check):
    """Who takes the division: the limits, zeros, subnormals, infinities, NaN."""
    e = np.nextafter
    b = np.array([2.0 ** -999, e(2.0 ** -999, 0.0), 2.0 ** 501, e(2.0 ** 501, 0.0), 0.0, -0.0,
                  5e-324, 1e-310, np.inf, -np.inf, np.nan, 1.7e308])
    assert check.far(0, b).tolist() == [False, True, True, False] + [True] * 8
    f = np.float32
    b32 = np.array([f(2.0 ** -111), e(f(2.0 ** -111), f(0)), f(2.0 ** 63), e(f(2.0 ** 63), f(0)),
                    f(0), f(1e-45), f(1e-40), f(np.inf), f(np.nan), f(3e38)], dtype=f)
    assert check.far(1, b32).tolist() == [False, True, True, False] + [True] * 6
    for op, v in ((RCP, b), (QUOTIENT, b), (QUOTIENT32, b32.astype(float))):
        got, want = check(op, 1.0, v)
        far = check.far(int(op == QUOTIENT32), v)
        assert np.array_equal(got[far], want[far], equal_nan=True)


def test_means_of_permeabilities(check):
    """The harmonic means' own operands, 2ab / (a + b), over forty decades."""
    rng = np.random.default_rng(4)
    for spread in (1.0, 10.0, 20.0):
        a, b = (10.0 ** rng.uniform(-spread, spread, N) for _ in range(2))
        got, want = check(QUOTIENT, 2.0 * a * b, a + b)
        _within(got, want, a + b, False)
        a, b = (v.astype(np.float32) for v in (a, b))
        with np.errstate(over="ignore"):
            use = (a * b > 0) & np.isfinite(2 * a * b)
        num, den = (2 * a[use] * b[use]).astype(float), (a[use] + b[use]).astype(float)
        got, want = check(QUOTIENT32, num, den)
        _within(got, want, den, True)
