"""Physics.__call__, whose step writes the tendencies anew, against the
pre-step's zeroing, the step that adds to the tendencies and the update, call
by call: bit-identical in every field, with one set of strides and with a
field of its own, in the modes that set or skip tendencies."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _physics(cfg, precision, own_strides):
    import torch

    from pyshield_b200.grid import GridData, GridIndexing, QuantityFactory, StencilFactory
    from pyshield_b200.inputs import PHYSICS_3D, PHYSICS_INTERFACE, PTOP, make_physics_state
    from pyshield_b200.physics import Physics, PhysicsState
    from pyshield_b200.quantity import Quantity

    nx, ny, L, h = 13, 9, 79, 3
    st, area = make_physics_state(nx, ny, L, seed=4, halo=h)
    gi = GridIndexing(nx, ny, L, h)
    qf = QuantityFactory(gi)

    def dev(a):
        t = torch.from_numpy(np.ascontiguousarray(a.transpose(tuple(reversed(range(a.ndim)))))).cuda()
        return t.permute(*reversed(range(a.ndim)))

    q = {}
    for nm in PHYSICS_3D:
        zi = nm in PHYSICS_INTERFACE
        a = dev(st[nm])
        if own_strides and nm == "qsnow":
            a = a.contiguous()  # k fastest
        q[nm] = Quantity(a, ("x", "y", "z_interface" if zi else "z"), "", (h, h, 0), (nx, ny, L + zi))
    q["land"] = Quantity(dev(st["land"]), ("x", "y"), "", (h, h), (nx, ny))
    ps = PhysicsState(**q, quantity_factory=qf, schemes=cfg.schemes)
    ar = np.zeros(st["land"].shape)
    ar[h:h + nx, h:h + ny] = area.reshape(ny, nx).T
    gd = GridData(Quantity(dev(ar), ("x", "y"), "", (h, h), (nx, ny)), PTOP)
    return Physics(StencilFactory(gi), qf, gd, cfg, precision=precision), ps, PHYSICS_3D


@pytest.mark.parametrize("own_strides", [False, True])
@pytest.mark.parametrize("precision,options", [
    ("plain", {}), ("mixed", {}), ("plain", {"sedi_transport": False, "do_qa": True, "do_sedi_w": False}),
])
def test_equals_the_separate_calls(precision, options, own_strides):
    import torch

    from pyshield_b200._config import PhysicsConfig
    from pyshield_b200.coupling import update_physics_state_with_tendencies
    from pyshield_b200.inputs import TENDENCY_FIELDS

    got = []
    for separate in (False, True):
        physics, ps, names = _physics(PhysicsConfig(dt_atmos=150.0, **options), precision, own_strides)
        for t in TENDENCY_FIELDS:  # stale values the step must not see
            getattr(ps.microphysics, t).view.fill_(float("nan"))
        if own_strides:
            t = ps.microphysics.qs_dt
            t.data = t.data.contiguous()  # k fastest
        m = ps.microphysics
        for _ in range(2):
            if not separate:
                physics(ps, 150.0)
                continue
            physics.prestep(ps)
            physics._microphysics(m, 150.0)
            update_physics_state_with_tendencies(
                ps.qvapor, ps.qliquid, ps.qrain, ps.qice, ps.qsnow, ps.qgraupel, ps.qcld, ps.pt, ps.ua, ps.va,
                m.qv_dt, m.ql_dt, m.qr_dt, m.qi_dt, m.qs_dt, m.qg_dt, m.qa_dt, m.pt_dt, m.udt, m.vdt,
                ps.physics_updated_specific_humidity, ps.physics_updated_qliquid, ps.physics_updated_qrain,
                ps.physics_updated_qice, ps.physics_updated_qsnow, ps.physics_updated_qgraupel,
                ps.physics_updated_cloud_fraction, ps.physics_updated_pt, ps.physics_updated_ua,
                ps.physics_updated_va, 150.0)
        got.append({n: getattr(ps, n).data.clone() for n in names}
                   | {t: getattr(ps.microphysics, t).data.clone() for t in TENDENCY_FIELDS})
    for n in got[0]:
        assert torch.equal(got[0][n], got[1][n]), n
