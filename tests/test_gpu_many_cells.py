"""Single-member wavefronts with several cells per thread that wait for outflows: the
same bits as with a grid barrier per step (a mask that leaves no cell out), whatever
the launches' lengths."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,temp", [("fp64", False), ("fp64", True), ("fp32", False)])
@pytest.mark.parametrize("kd,chunk", [(1, 0), (1, 100), (2, 7), (5, 0)])
def test_same_bits_as_a_grid_barrier(precision, temp, kd, chunk):
    from watergap2_gb300 import synthetic as sy
    from watergap2_gb300.gpu import Model
    region, nd = sy.region_small_swb(seed=5, ny=17, nx=31, river_velo_opt=2), 150
    P, T, S = sy.forcing(region, nd, seed=4, doy0=330)
    got = []
    for mask in (False, True):
        m = Model(region, max_days=nd, days_per_step=kd, precision=precision, water_temp=temp,
                  stations=np.arange(region.ncell))
        m.launch_shape(64, 3)   # 192 threads for 289 cells: a second cell for some lanes of the last warp
        if temp:
            m.set_water_temp_inputs(np.full(region.ncell, 9., np.float32))
            m.upload_longwave(0, 250. + T)
        m.upload_forcing(0, P, T, S)
        if mask:
            m.set_active_cells(np.ones(region.ncell))
        if chunk:
            m.chunk_steps(chunk)
        total = m.num_steps(nd)
        m.run_steps(330, 0, nd, 0, total // 2)
        m.run_steps(330, 0, nd, total // 2, total)
        s = m.get_state()
        got.append([m.discharge(0, nd)] + [np.asarray(s[k]) for k in sorted(s)] + ([*m.water_temp()] if temp else []))
    assert np.isfinite(got[0][0]).all() and got[0][0].max() > 0
    for a, b in zip(*got):
        assert np.array_equal(a, b)


def test_long_steps_share_launches():
    """Steps of 31 days: eight to a launch, not one."""
    from watergap2_gb300 import synthetic as sy
    from watergap2_gb300.gpu import Model
    region, nd = sy.region_64x64(size=9), 31 * 40
    P, T, S = sy.forcing(region, nd, seed=4)
    m = Model(region, max_days=nd, days_per_step=31, precision="fp32")
    m.upload_forcing(0, P, T, S)
    total, before = m.num_steps(nd), m.launch_count
    m.run_steps(1, 0, nd, 0, total)
    m.synchronize()
    assert total >= 40 and m.launch_count - before <= 2 * -(-total // 8)


@pytest.mark.parametrize("members", [1, 3])
def test_long_runs_that_gain_nothing_from_longer_steps_take_days(members):
    """As many launches with up to four days per step as with one."""
    from watergap2_gb300 import synthetic as sy
    from watergap2_gb300.gpu import Model
    region, nd = sy.region_64x64(size=9), 1460
    P, T, S = sy.forcing(region, nd, seed=4)
    launches = []
    for kd in (1, 4):
        m = Model(region, max_days=nd, days_per_step=kd, precision="fp32", members=members)
        m.upload_forcing(0, P, T, S)
        m.chunk_steps(16 // kd)
        before = m.launch_count
        m.run_days(1, 0, nd)
        m.synchronize()
        launches.append(m.launch_count - before)
    assert launches[0] == launches[1]
