"""Physics without the microphysics scheme needs nothing of the namelist but
its schemes."""
import types

from pyshield_b200.grid import GridData, GridIndexing, QuantityFactory, StencilFactory
from pyshield_b200.physics import Physics


def test_namelist_of_schemes_alone():
    gi = GridIndexing(4, 3, 5)
    physics = Physics(StencilFactory(gi), QuantityFactory(gi, device="cpu"), GridData(None, ptop=100.0),
                      types.SimpleNamespace(schemes=[]))
    assert not physics._gfs_microphysics
