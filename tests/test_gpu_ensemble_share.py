"""Ensembles that fill the GPU: the wavefront whose warps take a block's states from a
counter gives the same bits as the plain mapping of states to threads."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("what,members", [("bodies", 541), ("plain", 70)])   # members: not a whole number of warps
@pytest.mark.parametrize("kd,chunk", [(1, 0), (5, 3)])
def test_same_bits_as_the_plain_mapping(what, members, kd, chunk):
    from watergap2_gb300 import synthetic as sy
    from watergap2_gb300.gpu import Model
    region = sy.region_small_swb(seed=5, ny=17, nx=31) if what == "bodies" else sy.region_64x64(size=48)
    nd = 23
    P, T, S = sy.forcing(region, nd, seed=4, doy0=80)
    rng = np.random.default_rng(2)
    pf, gf = rng.uniform(0.8, 1.2, members), rng.uniform(0.5, 2.0, members)
    assert region.ncell * members >= 152 * 1024   # a state for every thread of the device
    got = []
    for shape in (None, 300):
        m = Model(region, max_days=nd, precision="fp32", members=members, prec_factor=pf, gamma_factor=gf,
                  days_per_step=kd, stations=np.arange(region.ncell, dtype=np.int32))
        if shape:
            m.launch_shape(64, shape)
        m.upload_forcing(0, P, T, S)
        if chunk:
            m.chunk_steps(chunk)
        total = m.num_steps(nd)
        m.run_steps(80, 0, nd, 0, total // 2)
        m.run_steps(80, 0, nd, total // 2, total)
        states = [m.get_state(k) for k in (0, members // 2, members - 1)]
        got.append([m.discharge(0, nd)] + [np.asarray(s[f]) for s in states for f in sorted(s)])
    assert np.isfinite(got[0][0]).all() and got[0][0].max() > 0
    for a, b in zip(*got):
        assert np.array_equal(a, b)
