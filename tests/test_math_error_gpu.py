"""The device's exponential, logarithm, powers and saturation humidities lose
no more than the functions they replace (CUDA's exp, log and pow, and the
reference's expressions of them): over each range of arguments that the step
meets, against extended precision, neither the largest error nor the mean
square exceeds CUDA's on the same arguments.

A result within 0.51 units in the last place counts as correctly rounded, and
mean squares that differ by less than 0.2 % as equal: a correctly rounded
result has 0.5 and 0.2887 units by itself, and two such functions differ by
that much over a million arguments (the mean square of N uniform errors
scatters by 0.9 / sqrt(N))."""
import numpy as np
import pytest

from test_math_gpu import EXP, LD, LOG, POW, QSI, QSI_DT, QSW, QSW_DT, device, ulps

pytestmark = pytest.mark.gpu

CUDA_EXP, CUDA_LOG, CUDA_POW, CUDA_EXP_LOG = 9, 10, 11, 16
CUDA_QS = {QSW: 12, QSW_DT: 13, QSI: 14, QSI_DT: 15}
N = 1_000_000


def mantissas(rng, lo, hi):
    """Numbers between lo and hi, uniform in each binade. (Exponentials of
    uniform numbers would have logarithms next to doubles.)"""
    x = np.ldexp(rng.uniform(1.0, 2.0, N), rng.integers(np.floor(np.log2(lo)), np.ceil(np.log2(hi)), N))
    return x[(x >= lo) & (x <= hi)]


def compare(fn, cuda, x, y, exact, what):
    stats = []
    for f in (fn, cuda):
        u = ulps(device(f, x, y), exact).astype(float)
        stats.append((u.max(), np.sqrt(np.mean(u**2))))
    (worst, rms), (cuda_worst, cuda_rms) = stats
    print(f"{what}: {worst:.4f} (rms {rms:.4f}), CUDA {cuda_worst:.4f} ({cuda_rms:.4f})")
    assert worst <= max(0.51, cuda_worst)
    assert rms <= 1.002 * cuda_rms


@pytest.mark.parametrize("lo,hi", [(-0.35, 0.35), (-3.0, 3.0), (-25.0, 5.0), (-60.0, 60.0), (-699.0, 699.0)])
def test_exp(lo, hi):
    x = np.random.default_rng(1).uniform(lo, hi, N)
    compare(EXP, CUDA_EXP, x, None, np.exp(LD(x)), f"exp [{lo}, {hi}]")


@pytest.mark.parametrize("lo,hi", [(1e-14, 1.0), (1e-9, 1e-2), (0.5, 2.0), (0.7, 1.42), (0.9, 1.1), (1e-300, 1e300)])
def test_log(lo, hi):
    x = mantissas(np.random.default_rng(2), lo, hi)
    compare(LOG, CUDA_LOG, x, None, np.log(LD(x)), f"log [{lo}, {hi}]")


@pytest.mark.parametrize("c,replaced", [
    # the reference's powers: density and mixing ratio, air's density, CCN
    (0.65625, "CUDA_POW"), (0.6875, "CUDA_POW"), (0.25, "CUDA_POW"), (-1.0 / 3.0, "CUDA_POW"),
    # those it writes as exp(c log x)
    (0.0625, "CUDA_EXP_LOG"), (0.2, "CUDA_EXP_LOG"), (0.65625, "CUDA_EXP_LOG"), (0.725, "CUDA_EXP_LOG"),
    (0.8125, "CUDA_EXP_LOG"), (0.875, "CUDA_EXP_LOG"), (0.95, "CUDA_EXP_LOG"), (1.75, "CUDA_EXP_LOG"),
    (7.0 / 3.0, "CUDA_EXP_LOG")])
def test_power(c, replaced):
    x = mantissas(np.random.default_rng(3), 1e-14, 1e10 if c < 0.0 else 10.0)
    compare(POW, globals()[replaced], x, c, np.power(LD(x), LD(c)), f"power {c:.4f}")


@pytest.mark.parametrize("ice", [False, True])
@pytest.mark.parametrize("lo,hi", [(170.0, 330.0), (200.0, 273.15), (273.2, 310.0), (150.1, 398.9)])
def test_saturation_humidity(lo, hi, ice):
    from pyshield_b200 import constants as C

    rng = np.random.default_rng(4)
    t, den = rng.uniform(lo, hi, N), np.exp(rng.uniform(np.log(1e-3), np.log(2.0), N))
    cold = ice & (t < C.TICE)
    dc, lh = np.where(cold, LD(C.D2ICE), LD(C.DC_VAP)), np.where(cold, LD(C.LI2), LD(C.LV0))
    t0, rv = LD(C.TICE), LD(C.RVGAS)
    te = np.minimum(LD(t), t0 + 102) if ice else LD(t)
    q = LD(C.E00) * np.exp((dc * np.log(te / t0) + lh * (te - t0) / (te * t0)) / rv) / (rv * te * LD(den))
    for fn, exact in ((QSI if ice else QSW, q), (QSI_DT if ice else QSW_DT, q * (dc + lh / te) / (rv * te))):
        stats = []
        for f in (fn, CUDA_QS[fn]):
            err = np.abs(LD(device(f, t, den)) / exact - 1).astype(float)
            stats.append((err.max(), np.sqrt(np.mean(err**2))))
        (worst, rms), (ref_worst, ref_rms) = stats
        print(f"{'ice' if ice else 'water'} {fn} [{lo}, {hi}]: {worst:.2e} ({rms:.2e}), "
              f"reference {ref_worst:.2e} ({ref_rms:.2e})")
        assert worst <= ref_worst and rms <= ref_rms
