"""Inputs that are not finite, or next to nothing, where one operation now stands for
several: what the reference's expressions keep finite stays finite."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_infinite_precipitation_on_snow():
    """All of it falls as snow: none reaches the soil."""
    from oracle import Oracle
    from watergap2_gb300 import synthetic as sy
    from watergap2_gb300.gpu import Model
    region, nd = sy.region_64x64(size=9), 6
    P, T, S = sy.forcing(region, nd, seed=4, doy0=340)
    T[:] = -40.
    P[2, 40] = np.inf
    m = Model(region, max_days=nd, stations=np.arange(region.ncell))
    q = m.run(340, P, T, S)
    o = Oracle(region)
    ref, _ = o.run(340, P, T, S, discharge=True)
    assert np.isfinite(ref).all() and np.isfinite(q).all()
    got, want = m.get_state(), o.state
    assert np.isinf(want["snow"][40]) and np.isfinite(want["soil"]).all()
    for k in ("canopy", "soil", "snow", "gw", "river"):
        assert np.allclose(got[k], want[k], rtol=1e-10, atol=1e-12)
