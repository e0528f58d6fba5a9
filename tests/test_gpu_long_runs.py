"""Runs longer than one launch's grid holds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_evaporation_of_more_days_than_a_grid_holds():
    from watergap2_gb300 import synthetic as sy
    from watergap2_gb300.gpu import Model
    region, nd = sy.region_64x64(size=3), 65535 * 8 + 1000
    P, T, S = sy.forcing(region, 365, seed=4)
    W = [np.resize(x, (nd, region.ncell)) for x in (P, T, S)]
    q = []
    for ring in (0, 4096):   # all days' evaporation at once, and in pieces
        m = Model(region, max_days=nd, ring_days=ring)
        m.upload_forcing(0, *W)
        m.run_days(1, 0, nd)
        q.append(m.discharge(nd - 365, 365))
        m.close()
    assert q[0].max() > 0 and np.array_equal(*q)


def test_the_ring_holds_as_many_days_as_its_memory():
    """8 GB of runoff and recharge; a launch may take half of them."""
    from watergap2_gb300 import synthetic as sy
    from watergap2_gb300.gpu import Model
    m = Model(sy.region_64x64(), max_days=100_000)
    assert m.vertical_overlap() > 0
    assert m.chunk_steps(50_000) == 50_000
