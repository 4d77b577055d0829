"""A tendency storage that the step cannot take is refused before the physics
step changes anything."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spoil", ["dtype", "host", "shape"])
@pytest.mark.parametrize("de_ice", [False, True])
def test_state_unchanged(spoil, de_ice):
    import torch

    from pyshield_b200._config import PhysicsConfig

    from test_physics_fresh_gpu import _physics

    physics, ps, names = _physics(PhysicsConfig(dt_atmos=150.0, de_ice=de_ice), "plain", False)
    t = ps.microphysics.qs_dt
    t.data = {"dtype": t.data.float(), "host": t.data.cpu(), "shape": t.data[:10]}[spoil]
    before = {n: getattr(ps, n).data.clone() for n in names}
    with pytest.raises((TypeError, ValueError)):
        physics(ps, 150.0)
    for n in names:
        assert torch.equal(getattr(ps, n).data, before[n]), n
