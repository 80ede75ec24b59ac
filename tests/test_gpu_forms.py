"""The sweeps' own quotients, roots and powers on the device (mdg_hydro.cuh, mdg_mixed.cuh),
against the exact values; where FP32 has no number for a face's wave speeds, against the FP64
solver."""
import itertools

import numpy as np
import pytest

from medusa_b200 import problems as P
from medusa_b200.solver import PREC_FP64, PREC_MIXED, Solver
from tests import _device

pytestmark = pytest.mark.gpu

N = 400000
EDGES64 = np.array([0.0, np.inf, np.nan, 1.0, 3.7, 1.0e-300, 1.0e-200, 1.0e-160, 1.0e160, 1.0e200, 1.0e300])


def _wide(rng, n, lo, hi, dtype):
    return ((1.0 + rng.random(n)) * 2.0 ** rng.integers(lo, hi, n)).astype(dtype)


def _ulps(got, want):
    """Error in units of the last place of `want` (which is held in a wider type)."""
    near = np.abs(want).astype(got.dtype)
    return float(np.max(np.abs(got.astype(want.dtype) - want) / np.spacing(near).astype(want.dtype)))


def _same(got, want, ulps):
    ok = (np.isnan(got) & np.isnan(want)) | (got == want)
    with np.errstate(invalid="ignore", over="ignore"):
        near = np.isfinite(want) & (np.abs(got - want) <= ulps * np.spacing(np.abs(want)))
    assert np.all(ok | near), [(g, w) for g, w in zip(got[~(ok | near)], want[~(ok | near)])]


def test_fp32_quotient_and_root():
    # one correction of an estimate of 2^-22: half an ulp, and 2^-20 of one, where the remainder (2^-23
    # of the numerator or radicand) is a normal number or nearly; below that the estimate alone
    rng = np.random.default_rng(1)
    for lo, bar in ((-60, 0.501), (-126, 2.0)):
        a, b = _wide(rng, N, lo, lo + 100, np.float32), _wide(rng, N, -25, 25, np.float32)
        want = a.astype(np.float64) / b.astype(np.float64)
        ok = want >= 2.0 ** -126
        assert _ulps(_device.form(0, a, b)[ok], want[ok]) <= bar
        assert _ulps(_device.form(1, a, a), np.sqrt(a.astype(np.float64))) <= bar


def test_mixed_faces_beside_cold_gas():
    """A pressure down to FP32's smallest subnormal number, beside gas of pressure one: a face that the mixed solver accepts has FP64's signal speed (which limits dt) and flux; where a
    wave speed is no number in FP32 it declines."""
    cold = [1.0e-45, 3.0e-44, 1.0e-42, 1.0e-39, 2.0e-38, 1.0e-36, 1.0e-20, 1.0e-6]
    v = [-30.0, -3.0, 0.0, 3.0, 30.0]
    st = [((1.0, a, p), (r, b, 1.0)) for p in cold for a in v for b in v for r in (0.1, 1.0, 10.0)]
    st = np.array(st + [(y, x) for x, y in st])
    for gam in (4.0 / 3.0, 5.0 / 3.0):
        o = _device.faces(gam, st)
        ok = o[:, 0] == 1.0
        assert 0.1 < np.mean(ok) < 1.0
        assert np.max(np.abs(o[ok, 1] - o[ok, 2]) / o[ok, 2]) <= 1.0e-4
        scale = np.max(np.abs(o[ok, 8:]), axis=1, keepdims=True)
        assert np.max(np.abs(o[ok, 3:8] - o[ok, 8:]) / scale) <= 1.0e-3


def test_fp32_power_of_the_wave_speeds():
    # powf's bound; the exponents are (G-1)/2G and 2G/(G-1) of the adiabatic indices
    rng = np.random.default_rng(2)
    x = np.exp(rng.uniform(-12.0, 12.0, N)).astype(np.float32)
    for g in (4.0 / 3.0, 1.4, 5.0 / 3.0, 2.0):
        for y in ((g - 1.0) / (2.0 * g), 2.0 * g / (g - 1.0)):
            y32 = np.full(N, y, dtype=np.float32)
            want = np.power(x.astype(np.float64), y32.astype(np.float64))
            ok = (want < 1.0e38) & (want > 1.0e-37)
            assert _ulps(_device.form(2, x, y32)[ok], want[ok]) <= 4.0


def test_fp64_reciprocals_and_sound_speed():
    # two Newton steps from 2^-20: the roundings of the last one (rsqrt: of its product too)
    rng = np.random.default_rng(3)
    b, c = _wide(rng, N, -300, 300, np.float64), _wide(rng, N, -300, 300, np.float64)
    wide = lambda v: v.astype(np.longdouble)
    assert _ulps(_device.form(0, b, b), 1 / wide(b)) <= 1.0
    assert _ulps(_device.form(1, b, b), 1 / np.sqrt(wide(b))) <= 1.5
    assert _ulps(_device.form(2, b, c), np.sqrt(wide(b) / wide(c))) <= 2.5


def test_fp64_sound_speed_at_the_edges():
    with np.errstate(all="ignore"):
        pairs = np.array(list(itertools.product(EDGES64, EDGES64)))
        q = pairs[:, 0] / pairs[:, 1]
        lost = np.all(np.isfinite(pairs) & (pairs > 0.0), axis=1) & ~((q > 1.0e-307) & (q < np.inf))
        got = _device.form(2, pairs[:, 0], pairs[:, 1])
        _same(got[~lost], np.sqrt(q[~lost]), 2.5)   # (elsewhere the operators' quotient is no number)


@pytest.mark.parametrize("mixed", [False, True])
def test_fp64_quotients_by_one_reciprocal(mixed):
    """Plain FP64: the division's bits, whatever the numbers; the mixed sweeps' form: the roundings
    of the reciprocal and of the product."""
    rng = np.random.default_rng(4)
    a = _wide(rng, 5 * N, -200, 200, np.float64) * np.where(rng.random(5 * N) < 0.5, -1.0, 1.0)
    b = _wide(rng, N, -200, 200, np.float64)
    q = np.nextafter(2.0 ** rng.integers(-9, 9, N // 4), 0.0)      # divisors next below a power of two
    b[:N // 4] = q
    if not mixed:
        e = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 1.0, 5.0e-324, 1.0e-310, 1.0e-200, 1.7e308])
        k = rng.integers(0, 5 * N, 20000)
        a[k] = e[rng.integers(0, e.size, k.size)]
        k = rng.integers(0, N, 4000)
        b[k] = e[rng.integers(0, e.size, k.size)]
    got = _device.form(4 if mixed else 3, a, b)
    with np.errstate(all="ignore"):
        want = a / np.repeat(b, 5)
    if mixed:
        assert np.all(np.abs(got - want) <= 2.0 * np.spacing(np.abs(want)))
    else:
        assert np.array_equal(got, want, equal_nan=True)
        assert np.array_equal(np.signbit(got) | np.isnan(got), np.signbit(want) | np.isnan(want))


def _mixed_errors(batches, steps):
    """Geometric mean over all problems of the mixed sweep's relative error (2-norm) of density and
    internal energy against the plain FP64 sweep after the same steps."""
    e = []
    for pbs in batches:
        state = []
        for prec in (PREC_FP64, PREC_MIXED):
            with Solver(pbs, precision=prec) as s:
                s.step(steps)
                s.synchronize()
                state.append([s.update_cpu(m) for m in range(len(pbs))])
        for a, b in zip(*state):
            e.append([np.linalg.norm(b[:, v] - a[:, v]) / np.linalg.norm(a[:, v]) for v in (0, 1)])
    return np.exp(np.mean(np.log(np.array(e) + 1.0e-18), axis=0))


# What the sweeps had with correctly rounded quotients and roots, without contraction: (density,
# internal energy).  Over such samples the means of two builds differ by up to a tenth, so a bar of 1.25.
ROUNDED = {"ensemble": (1.670e-8, 3.911e-8), "shear": (1.233e-8, 1.992e-8), "blast2d": (2.650e-9, 1.785e-8),
           "blast3d": (2.105e-9, 8.992e-9)}
SAMPLES = {
    "ensemble": (lambda: [P.ensemble_1d(96, seed=21, nmin=100, nmax=2000)], 40),
    "shear": (lambda: [[P.kelvin_helmholtz(70 + 53 * i, 60 + 61 * (i * 5 % 8))] for i in range(6)], 60),
    "blast2d": (lambda: [[P.sedov_2d_spherical(80 + 37 * i, (32, 64, 128)[i % 3], noise=0.01, r_dep=0.05)]
                         for i in range(6)], 60),
    "blast3d": (lambda: [[P.sedov_3d(50 + 11 * i, (16, 32)[i % 2], (32, 64)[i % 2], noise=0.01, r_dep=0.1)]
                         for i in range(6)], 60),
}


@pytest.mark.parametrize("kind", sorted(SAMPLES))
def test_mixed_sweeps_are_as_near_to_fp64_as_with_rounded_operations(kind):
    make, steps = SAMPLES[kind]
    got = _mixed_errors(make(), steps)
    assert np.all(got <= 1.25 * np.array(ROUNDED[kind])), got
