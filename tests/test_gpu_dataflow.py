"""The wavefront whose steps wait for the upstream outflows themselves: the same
bits as the one with per-warp step flags, at the edges of its launches (one step,
the whole buffer, split runs) and of its warps (one cell, a partial warp, classes
of water bodies that fill less than a warp); the per-day call's waits run out like
the grid barrier's; states read on the device in cell order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _state(m):
    s = m.get_state()
    return np.concatenate([np.asarray(s[k], np.float64).ravel() for k in sorted(s)])


def _region(what):
    from watergap2_gb300 import synthetic as sy
    return {"one warp": lambda: sy.region_64x64(size=5), "partial": lambda: sy.region_64x64(size=9),
            "bodies": lambda: sy.region_small_swb(seed=5, ny=17, nx=31, river_velo_opt=2)}[what]()


@pytest.mark.parametrize("what", ["one warp", "partial", "bodies"])
@pytest.mark.parametrize("kd,chunk", [(1, 0), (1, 1), (1, 64), (5, 3), (31, 1)])
def test_same_bits_as_step_flags(what, kd, chunk):
    from watergap2_gb300 import synthetic as sy
    from watergap2_gb300.gpu import Model
    region, nd = _region(what), 70
    P, T, S = sy.forcing(region, nd, seed=4, doy0=330)
    got = []
    for flags in (1, 0):
        m = Model(region, max_days=nd, days_per_step=kd, stations=np.arange(region.ncell))
        m.step_sync(flags)
        m.vertical_overlap(not flags)
        m.upload_forcing(0, P, T, S)
        if not flags and chunk <= (nd // kd) // 2:
            m.chunk_steps(chunk)
        total = m.num_steps(nd)
        m.run_steps(330, 0, nd, 0, total // 3)       # the wavefront goes on across calls
        m.run_steps(330, 0, nd, total // 3, total)
        q1 = m.discharge(0, nd)
        m.run_days(330, 0, nd)                       # and with its own choice of days per step
        got.append((q1, m.discharge(0, nd), _state(m)))
    for a, b in zip(*got):
        assert np.array_equal(a, b)


def test_per_day_waits_run_out_and_the_context_recovers():
    from watergap2_gb300 import synthetic as sy
    from watergap2_gb300.gpu import Model, WgError
    region = _region("bodies")
    P, T, S = sy.forcing(region, 3, seed=4)
    ref = Model(region, max_days=3, stations=np.arange(region.ncell)).run(1, P, T, S, per_day=True)
    m = Model(region, max_days=3, stations=np.arange(region.ncell))
    m.upload_forcing(0, P, T, S)
    m.save_snapshot()
    m.barrier_test(1)
    m.step_vertical(1, 0)
    m.step_routing(1, 0)
    with pytest.raises(WgError, match="device wait exceeded its limit"):
        m.synchronize()
    m.barrier_test(0)
    m.clear_error()
    m.restore_snapshot()
    assert np.array_equal(m.run(1, P, T, S, per_day=True), ref)


@pytest.mark.parametrize("nband,members", [(1, 1), (5, 1), (30, 1), (31, 1), (40, 1), (5, 3)])
def test_state_reads_in_cell_order(nband, members):
    from watergap2_gb300 import synthetic as sy
    from watergap2_gb300.gpu import Model
    region = sy.region_64x64(size=9, nband=nband)
    m = Model(region, max_days=2, precision="fp32" if members > 1 else "fp64", members=members)
    rng = np.random.default_rng(3)
    want = []
    for k in range(members):
        st = m.get_state(member=k)
        for name, a in st.items():
            st[name] = rng.integers(0, 99, a.shape).astype(a.dtype) if a.dtype == np.int32 \
                else rng.random(a.shape).astype(np.float32).astype(np.float64)
        m.set_state(st, member=k)
        want.append(st)
    for k in range(members):
        got = m.get_state(member=k)
        assert all(np.array_equal(got[name], want[k][name]) for name in got)
        some = m.get_state(member=k, fields=("soil", "snow_band", "lai_days"))
        assert all(np.array_equal(some[name], want[k][name]) for name in some)
