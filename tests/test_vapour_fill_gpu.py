"""UpdateAtmosphereState's vapour fill over blocks that need it and blocks that
do not: the launch leaves the sweeps out for 32 consecutive columns without a
level that they would change. Bit for bit the oracle's fill_gfs_delp, with
deficits in a few columns: at either end of the column, in runs, at values next
to the limits (1e-9; zero at the top level)."""
import types

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PATTERNS = [
    {0: -1e-7}, {0: -0.0}, {0: 5e-10}, {1: 5e-10}, {1: -1e-6}, {0: -1e-6, 1: -2e-6}, {"mid": 0.0},
    {"mid": np.nextafter(1e-9, 0.0)}, {"mid": 1e-9}, {"last": -1e-5}, {"last": 1e-10}, {"run": -3e-6}, {"all": -1e-8},
]


def _vapour(rng, ncol, L, needy):
    q = rng.uniform(2e-9, 2e-3, (ncol, L + 1))
    for n, c in enumerate(needy):
        for where, v in PATTERNS[n % len(PATTERNS)].items():
            k = {"mid": L // 2, "last": L - 1, "run": slice(L // 3, L // 3 + 5), "all": slice(0, L)}.get(where, where)
            q[c, k] = v
    return q


@pytest.mark.parametrize("own_strides", [False, True])
@pytest.mark.parametrize("L", [2, 3, 79, 128])
def test_fill(L, own_strides):
    import torch

    from oracle import coupling as OC
    from pyshield_b200._config import PhysicsConfig
    from pyshield_b200.coupling import UpdateAtmosphereState
    from pyshield_b200.grid import GridIndexing, StencilFactory
    from pyshield_b200.quantity import Quantity

    nx, ny, h = 43, 25, 3
    mx, my = nx + 2 * h, ny + 2 * h  # 1,519 columns: 48 blocks, the last one partly filled
    rng = np.random.default_rng(L)
    needy = [5, 32, 63, 64 + 31] + list(range(320, 320 + 3 * len(PATTERNS), 3)) + [mx * my - 1]
    q = np.zeros((mx + 1, my + 1, L + 1))
    q[:mx, :my] = _vapour(rng, mx * my, L, needy).reshape(my, mx, L + 1).transpose(1, 0, 2)
    delp = rng.uniform(50.0, 2000.0, q.shape)
    want = q.copy()
    OC.fill_gfs_delp(delp[:mx, :my], want[:mx, :my], 1.0e-9)

    def dev(a, kfast=False):
        t = torch.from_numpy(np.ascontiguousarray(a if kfast else a.T)).cuda()
        t = t if kfast else t.permute(*range(a.ndim)[::-1])
        return Quantity(t, ("x", "y", "z")[:a.ndim], "", (h, h, 0)[:a.ndim], (nx, ny, L)[:a.ndim])

    other = np.zeros_like(q)
    d = types.SimpleNamespace(**{k: dev(other) for k in ("qliquid", "qrain", "qsnow", "qice", "qgraupel", "pt", "pe",
                                                         "peln", "pk", "ua", "va")})
    d.qvapor, d.delp, d.ps = dev(q, own_strides), dev(delp), dev(other[..., 0])
    p = types.SimpleNamespace(**{"physics_updated_" + k: dev(other) for k in (
        "ua", "va", "pt", "specific_humidity", "qliquid", "qrain", "qsnow", "qice", "qgraupel")},
        ua=dev(other), va=dev(other), pt=dev(other), prsi=dev(other))
    uas = UpdateAtmosphereState(StencilFactory(GridIndexing(nx, ny, L, h)), None, PhysicsConfig(dt_atmos=150),
                                dycore_only=True)
    uas(d, p, dev(other), dev(other), dev(other), 150.0)
    got = d.qvapor.data.cpu().numpy()
    np.testing.assert_array_equal(got[:mx, :my, :L], want[:mx, :my, :L])
    np.testing.assert_array_equal(got[mx:], 0.0)
    np.testing.assert_array_equal(got[:, :, L], q[:, :, L])
