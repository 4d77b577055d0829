"""65 to 80 levels, two columns packed on a group of warps: a column's sums
associate by its slot, the group's first or second, and by nothing else. Every
column of every launch shape equals, bit for bit, the same column in the same
slot of the smallest shape: of a domain that starts with it in its own slot, or
of one shifted by a leading column."""
import numpy as np
import pytest

from golden_io import MP_TENDENCIES, PRECIP

pytestmark = pytest.mark.gpu

FIELDS = MP_TENDENCIES + ("wmp", "qaz") + PRECIP


@pytest.mark.parametrize("precision", ["plain", "mixed"])
@pytest.mark.parametrize("L", [65, 79, 80])
def test_both_slots(L, precision):
    from pyshield_b200._config import PhysicsConfig
    from pyshield_b200.inputs import make_state

    from mp_helpers import run_gpu

    n = 37  # odd: a repetition's columns change slots from one to the next
    state, area = make_state(n, L, seed=L, n_cube=12, sat_fraction=0.1)
    cfg = PhysicsConfig(dt_atmos=150.0)
    lead = {k: np.concatenate([v[..., -1:], v], axis=-1) for k, v in state.items()}
    ref = [run_gpu(cfg, state, area, n, 1, 150.0, precision=precision)[0],
           run_gpu(cfg, lead, np.concatenate([area[-1:], area]), n + 1, 1, 150.0, precision=precision)[0]]
    # just inside and beyond the domains of 2, 4, 6 and 8 columns per block (148 blocks a wave)
    for r in sorted({max(1, (g * 148) // n + d) for g in (2, 4, 6, 8) for d in (0, 1)}):
        big = {k: np.concatenate([v] * r, axis=-1) for k, v in state.items()}
        out = run_gpu(cfg, big, np.concatenate([area] * r), n, r, 150.0, precision=precision)[0]
        for f in FIELDS:
            got = out[f].reshape(out[f].shape[:-1] + (r, n))
            for slot, want in enumerate((ref[0][f], ref[1][f][..., 1:])):
                mine = got[..., slot::2, :]
                assert np.array_equal(mine, np.broadcast_to(want[..., None, :], mine.shape)), (f, r, slot)
