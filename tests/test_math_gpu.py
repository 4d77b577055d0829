"""Errors of the device's FP64 division, square root, exp, log, powers and
saturation humidities against extended precision (numpy longdouble, 64-bit
significand), over the ranges the step meets and at the edges where a form
changes: argument limits beyond which CUDA's function is called, the ends of
the fast saturation formula's temperatures, zero, infinity and NaN.

Tolerances, in units of the last place of the correctly rounded result:
a corrected quotient or root is half a unit but for the rare operand whose
residual rounds (0.51); exp and a power lose one rounding of the reduced
argument times at most 0.35 of the result, and the final one, each doubled
where the result lies in the lower half of its binade (2); a log has the
quotient, the series and the final sum (3, of a log no smaller than 1e-3).
A saturation humidity's exponent is two terms of at most 22 with three
roundings each (7.4e-15), then ten roundings (1.2e-15): 1e-14 relative."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LD = np.longdouble
DIV, SQRT, EXP, LOG, POW, QSW, QSW_DT, QSI, QSI_DT = range(9)
N = 20011


def device(fn, x, y=None):
    import torch

    from pyshield_b200.build import PROBE_LIB

    lib = ctypes.CDLL(PROBE_LIB)
    lib.shield_probe_math.argtypes = [ctypes.c_int, ctypes.c_int] + [ctypes.c_void_p] * 4
    a = torch.from_numpy(np.ascontiguousarray(x)).cuda()
    b = torch.from_numpy(np.broadcast_to(1.0 if y is None else y, x.shape).copy()).cuda()
    out = torch.empty_like(a)
    rc = lib.shield_probe_math(fn, a.numel(), a.data_ptr(), b.data_ptr(), out.data_ptr(),
                               torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    return out.cpu().numpy()


def ulps(got, exact):
    near = np.asarray(exact, dtype=np.float64)
    return np.abs(LD(got) - exact) / LD(np.spacing(np.abs(near)))


def logu(rng, lo, hi, n=N):
    return np.exp(rng.uniform(np.log(lo), np.log(hi), n))


@pytest.mark.parametrize("fn", [DIV, SQRT, EXP, LOG, POW])
def test_units_in_the_last_place(fn):
    rng = np.random.default_rng(fn)
    y = None
    if fn == DIV:
        x = rng.choice([-1.0, 1.0], N) * logu(rng, 1e-200, 1e60)
        y = rng.choice([-1.0, 1.0], N) * logu(rng, 1e-60, 1e60)
        exact, tol = LD(x) / LD(y), 0.51
    elif fn == SQRT:
        x = logu(rng, 1e-280, 1e280)
        exact, tol = np.sqrt(LD(x)), 0.51
    elif fn == EXP:
        x = np.concatenate([rng.uniform(-60.0, 60.0, N), rng.uniform(-708.0, 709.0, N), [700.0, -700.0, 0.0, 1e-300]])
        exact, tol = np.exp(LD(x)), 2.0
    elif fn == LOG:
        x = np.concatenate([logu(rng, 1e-40, 1e40), logu(rng, 2.3e-308, 1e308), 1.0 + rng.uniform(1e-3, 0.5, N),
                            [np.sqrt(0.5), np.sqrt(2.0), np.nextafter(np.sqrt(2.0), 2.0)]])
        exact, tol = np.log(LD(x)), 3.0
    else:
        x = np.concatenate([logu(rng, 1e-14, 1.0), logu(rng, 1e-20, 1e20)])
        y = rng.choice([0.0625, 0.2, 0.65625, 0.6875, 0.725, 0.8125, 0.875, 0.95, 1.75, 7.0 / 3.0, -1.0 / 3.0], 2 * N)
        exact, tol = np.power(LD(x), LD(y)), 2.0
    worst = float(ulps(device(fn, x, y), exact).max())
    print(f"function {fn}: {worst:.3f} ulp")
    assert worst <= tol


@pytest.mark.parametrize("fn,x,want", [
    (DIV, [0.0, -0.0], [0.0, -0.0]),
    (SQRT, [0.0, 2.2250738585072014e-308], [0.0, 1.4916681462400413e-154]),
    (EXP, [-np.inf, np.inf, -1e4, 1e4, -720.0], [0.0, np.inf, 0.0, np.inf, np.exp(-720.0)]),
    (LOG, [0.0, np.inf, 1.0, 5e-324], [-np.inf, np.inf, 0.0, np.log(5e-324)]),
    (POW, [0.0, 1.0, np.inf], [0.0, 1.0, np.inf]),
])
def test_special_values(fn, x, want):
    got = device(fn, np.array(x), np.array(0.5) if fn == POW else None)
    np.testing.assert_allclose(got, want, rtol=3e-15)
    assert np.isnan(device(fn, np.array([np.nan]))).all()
    if fn in (SQRT, LOG):
        assert np.isnan(device(fn, np.array([-1.0]))).all()


@pytest.mark.parametrize("ice", [False, True])
def test_saturation_humidity(ice):
    from pyshield_b200 import constants as C

    rng = np.random.default_rng(3)
    edges = np.array([113.16, 150.0, 273.16, 375.16, 399.0])
    t = np.concatenate([rng.uniform(170.0, 330.0, N), rng.uniform(100.0, 420.0, N), edges, np.nextafter(edges, 0.0),
                        np.nextafter(edges, 500.0)])
    den = logu(rng, 1e-3, 2.0, t.size)
    tl, dl, rv, t0 = LD(t), LD(den), LD(C.RVGAS), LD(C.TICE)
    dc = np.where(ice & (t < C.TICE), LD(C.D2ICE), LD(C.DC_VAP))
    lh = np.where(ice & (t < C.TICE), LD(C.LI2), LD(C.LV0))
    te = np.clip(tl, LD(C.T_SAT_MIN), t0 + 102) if ice else tl
    q = LD(C.E00) * np.exp((dc * np.log(te / t0) + lh * (te - t0) / (te * t0)) / rv) / (rv * te * dl)
    dq = q * (dc + lh / te) / (rv * te)
    for fn, exact in ((QSI if ice else QSW, q), (QSI_DT if ice else QSW_DT, dq)):
        # below 150 K the reference's own expression runs, whose exponent terms reach 40
        err = np.abs(LD(device(fn, t, den)) / exact - 1)
        near = (t > 150.0) & (t < 399.0)
        print(f"{'ice' if ice else 'water'} {fn}: {float(err[near].max()):.2e}, elsewhere {float(err[~near].max()):.2e}")
        assert float(err[near].max()) <= 1e-14
        assert float(err[~near].max()) <= 2e-14
