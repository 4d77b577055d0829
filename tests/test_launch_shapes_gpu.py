"""The step's launch choices do not change a column's result: its arithmetic
is the same whatever the number of columns per block (chosen from the domain's
size), and whether the staging forms one offset for all fields or one for
each. The plain form against the oracle is test_mp_gpu's; here the results
must be bit-identical."""
import numpy as np
import pytest

from golden_io import MP_TENDENCIES, PRECIP

pytestmark = pytest.mark.gpu

FIELDS = MP_TENDENCIES + ("wmp", "qaz") + PRECIP
# columns per block of each level range (csrc/mp_kernel.cuh, launch_shapes), 148 blocks in a wave
SHAPES = {31: (8, 24), 63: (4, 8, 12), 79: (2, 4, 6, 8), 90: (2, 4, 8), 127: (2, 4, 6, 7), 200: (1, 3)}


def _state(n, L):
    from pyshield_b200.inputs import make_state

    return make_state(n, L, seed=L, n_cube=12, sat_fraction=0.1)


@pytest.mark.parametrize("precision", ["plain", "mixed"])
@pytest.mark.parametrize("L", sorted(SHAPES))
def test_columns_per_block(L, precision):
    from pyshield_b200._config import PhysicsConfig

    from mp_helpers import run_gpu

    n = 37  # odd: the last block is partly filled
    state, area = _state(n, L)
    cfg = PhysicsConfig(dt_atmos=150.0)
    ref = run_gpu(cfg, state, area, n, 1, 150.0, precision=precision)[0]
    G = SHAPES[L]
    # a domain just inside and just beyond each wave limit, and far beyond the last
    reps = sorted({max(1, (g * 148) // n + d) for g in G for d in (0, 1)} | {8 * 7 * 148 // n + 1 if L == 127 else 1})
    for r in reps:
        big = {k: np.concatenate([v] * r, axis=-1) for k, v in state.items()}
        out = run_gpu(cfg, big, np.concatenate([area] * r), n, r, 150.0, precision=precision)[0]
        for f in FIELDS:
            got = out[f].reshape(out[f].shape[:-1] + (r, n))
            if 65 <= L <= 80:
                # a packed column's level sums associate by its slot (even or
                # odd column), as in one launch shape as in another
                got = got[..., ::2, :]
            assert np.array_equal(got, np.broadcast_to(ref[f][..., None, :], got.shape)), (f, r)


@pytest.mark.parametrize("precision", ["plain", "mixed"])
@pytest.mark.parametrize("odd", ["input", "tendency", "kfast"])
def test_fields_of_their_own_strides(odd, precision):
    """One field in a storage of another shape or memory order: the general staging."""
    import torch

    from pyshield_b200._config import PhysicsConfig
    from pyshield_b200.microphysics import Microphysics
    from pyshield_b200.quantity import Quantity

    from mp_helpers import device_state

    nx, ny, L = 11, 7, 79
    state, area = _state(nx * ny, L)
    outs = []
    for own in (False, True):
        ms, sf, qf, gd = device_state(state, area, nx, ny)
        if own:
            name = "qs_dt" if odd == "tendency" else "qsnow"
            v = getattr(ms, name).view
            shape = (nx, ny, L) if odd == "kfast" else (L + 2, ny + 1, nx + 3)
            t = torch.zeros(shape, dtype=torch.float64, device="cuda")
            t = t if odd == "kfast" else t.permute(2, 1, 0)
            t[:nx, :ny, :L] = v
            setattr(ms, name, Quantity(t, ("x", "y", "z"), "", (0, 0, 0), (nx, ny, L)))
        mp = Microphysics(sf, qf, gd, PhysicsConfig(dt_atmos=150.0), precision=precision)
        mp(ms, 150.0)
        outs.append([getattr(ms, f).view.clone() for f in MP_TENDENCIES + ("wmp",)] + [mp.rain.clone()])
    for a, b in zip(*outs):
        assert torch.equal(a, b)
