"""Ensembles that fill the GPU at every block size, and at the sizes where the vertical
balance ahead runs its denser variant."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [32, 64, 96, 128])
def test_block_sizes_give_the_same_bits(threads):
    """Joined blocks (the context's and the launch shape's) beside fewer, plain ones."""
    from watergap2_gb300 import synthetic as sy
    from watergap2_gb300.gpu import Model
    region, members, nd = sy.region_small_swb(seed=5, ny=17, nx=31), 541, 12
    assert region.ncell * members >= 152 * 1024   # a state for every thread of the device
    P, T, S = sy.forcing(region, nd, seed=4, doy0=80)
    pf = np.random.default_rng(2).uniform(0.8, 1.2, members)
    got = []
    for how in ("created", "shaped", "plain"):
        m = Model(region, max_days=nd, precision="fp32", members=members, prec_factor=pf,
                  block_threads=threads if how == "created" else 0, stations=np.arange(region.ncell, dtype=np.int32))
        if how != "created":
            m.launch_shape(threads, 300 if how == "plain" else 0)
        m.upload_forcing(0, P, T, S)
        m.run_days(80, 0, nd)
        s = m.get_state(members - 1)
        got.append([m.discharge(0, nd)] + [np.asarray(s[f]) for f in sorted(s)])
    assert np.isfinite(got[0][0]).all() and got[0][0].max() > 0
    for other in got[1:]:
        for a, b in zip(got[0], other):
            assert np.array_equal(a, b)


def test_denser_vertical_balance():
    """Eight states and more for every thread of the wavefront: the same bits as with
    the vertical balance on the second stream, which keeps the other variant, and as a
    single FP32 run."""
    from watergap2_gb300 import synthetic as sy
    from watergap2_gb300.gpu import Model
    region, members, nd = sy.region_64x64(size=48), 541, 4
    assert region.ncell * members >= 8 * 152 * 1024
    P, T, S = sy.forcing(region, nd, seed=4, doy0=340)
    pf = np.exp(np.random.default_rng(2).normal(0., 0.3, members)).astype(np.float32)
    pf[7] = 1.
    kw = dict(max_days=nd, precision="fp32", stations=np.arange(region.ncell, dtype=np.int32))
    got = []
    for overlap in (False, True):
        m = Model(region, members=members, prec_factor=pf, **kw)
        m.vertical_overlap(overlap)
        m.upload_forcing(0, P, T, S)
        m.run_days(340, 0, nd)
        s = [m.get_state(k) for k in (0, 7, members - 1)]
        got.append([m.discharge(0, nd)] + [np.asarray(x[f]) for x in s for f in sorted(x)])
    for a, b in zip(*got):
        assert np.array_equal(a, b)
    one = Model(region, **kw)
    q = one.run(340, P, T, S)
    assert q.max() > 0 and np.array_equal(m.member_discharge(7, 0, nd).reshape(q.shape), q)
    s = one.get_state()
    for f, b in zip(sorted(s), got[0][1 + len(s):1 + 2 * len(s)]):
        assert np.array_equal(np.asarray(s[f]), b)
