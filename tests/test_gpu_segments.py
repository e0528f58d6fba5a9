"""Parts of a run: steps t_begin > 0 from a graph, run again on the state they find, and
beside a change of what the steps wait for, against the step flags, whose calls keep
their outflows in the same two rows throughout."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
DOY0, ND = 330, 90


def _forcing(region):
    from watergap2_gb300 import synthetic as sy
    return sy.forcing(region, ND, seed=4, doy0=DOY0)


def _model(temp=False, flags=False, kd=1, **kw):
    from watergap2_gb300 import synthetic as sy
    from watergap2_gb300.gpu import Model
    region = sy.region_small_swb(seed=5, ny=17, nx=31, river_velo_opt=2)
    P, T, S = _forcing(region)
    m = Model(region, max_days=ND, days_per_step=kd, stations=np.arange(region.ncell), water_temp=temp, **kw)
    if temp:
        m.set_water_temp_inputs(np.full(region.ncell, 9., np.float32))
        m.upload_longwave(0, 250. + T)
    if flags:
        m.vertical_overlap(False)
        m.step_sync(1)
    m.upload_forcing(0, P, T, S)
    return m


def _all(m, temp):
    s = m.get_state()
    out = [m.discharge(0, ND)] + [np.asarray(s[k]) for k in sorted(s)]
    if temp:
        out += [*m.water_temp(), m.river_temp(0, ND)]
    return out


def _same(a, b):
    assert np.isfinite(a[0]).all() and a[0].max() > 0
    for x, y in zip(a, b):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("kd", [1, 5])
@pytest.mark.parametrize("temp", [False, True])
def test_graph_of_a_later_part(temp, kd):
    """Captured before the steps that lead to it have run, and before a graph of a
    whole run or a change of the waits would have told it anything."""
    ref = _model(temp, True, kd)
    total = ref.num_steps(ND)
    a, b = total // 4, total // 2
    ref.run_steps(DOY0, 0, ND, 0, total)
    m = _model(temp, False, kd)
    m.graph_capture(DOY0, 0, ND, a, b)
    m.run_steps(DOY0, 0, ND, 0, a)
    m.graph_launch()
    m.run_steps(DOY0, 0, ND, b, total)
    _same(_all(m, temp), _all(ref, temp))


@pytest.mark.parametrize("kd", [1, 5])
@pytest.mark.parametrize("temp", [False, True])
def test_steps_run_again(temp, kd):
    """A part longer than the rows of the waits, to the end of the run and into it."""
    got = []
    for flags in (True, False):
        m = _model(temp, flags, kd)
        total = m.num_steps(ND)
        m.run_steps(DOY0, 0, ND, 0, 20 // kd)
        m.save_snapshot()
        for end in (total, total - 3, total // 2):
            for _ in range(2):
                m.run_steps(DOY0, 0, ND, 20 // kd, end)
        out = _all(m, temp)
        m.restore_snapshot()
        if not flags:
            m.graph_capture(DOY0, 0, ND, 20 // kd, total)
        for _ in range(2):
            m.run_steps(DOY0, 0, ND, 20 // kd, total) if flags else m.graph_launch()
        got.append(out + _all(m, temp))
    _same(*got)


def test_waits_changed_between_the_steps():
    ref = _model(flags=True)
    total = ref.num_steps(ND)
    ref.run_steps(DOY0, 0, ND, 0, total)
    m = _model()
    cells = m.region.ncell
    cuts = [0, 1, 2, 7, 30, 31, 80, total]
    for k, (a, b) in enumerate(zip(cuts, cuts[1:])):
        m.step_sync(k % 3 == 1)
        m.set_active_cells(np.ones(cells) if k % 3 == 2 else None)
        m.run_steps(DOY0, 0, ND, a, b)
    _same(_all(m, False), _all(ref, False))


def test_autotune_on_later_steps_after_a_shorter_run():
    ref = _model(flags=True)
    ref.run_days(DOY0, 0, 40)
    m = _model()
    m.run_days(DOY0, 0, 40)
    m.autotune(DOY0, 0, ND, 70, 30)
    s, r = m.get_state(), ref.get_state()
    for k in s:
        assert np.array_equal(s[k], r[k])


def _above(region, x):
    """The cells above cell x."""
    up = np.zeros(region.ncell, bool)
    for i in region.rout_order[::-1]:
        d = region.downstream[i]
        up[i] = d >= 0 and (d == x or up[d])
    return up


def _cell_with_upstream(region):
    n = [_above(region, x).sum() for x in range(region.ncell)]
    return int(np.argsort(n)[-3])


@pytest.mark.parametrize("restored", [False, True])
def test_a_skipped_cell_has_no_outflow(restored):
    """Days routed before the mask leave nothing behind for the cells below it: as in
    the region whose river is cut there."""
    import copy
    from watergap2_gb300.gpu import Model
    m = _model()
    x = _cell_with_upstream(m.region)
    skip = _above(m.region, x)
    m.set_active_cells(np.ones(m.region.ncell))   # routed with a grid barrier per step
    m.run_days(DOY0, 0, 20)
    s = m.get_state()
    if restored:
        m.save_snapshot()
    m.set_active_cells(~skip)
    if restored:
        m.restore_snapshot()
    m.run_days((DOY0 - 1 + 20) % 365 + 1, 20, 30)

    cut = copy.deepcopy(m.region)
    cut.arrays["downstream"][skip & (cut.downstream == x)] = -1
    P, T, S = _forcing(m.region)
    r = Model(cut, max_days=ND, stations=np.arange(cut.ncell))
    r.upload_forcing(0, P, T, S)
    r.set_state(s)
    r.set_active_cells(~skip)
    r.run_days((DOY0 - 1 + 20) % 365 + 1, 20, 30)
    a, b = m.discharge(20, 30)[:, ~skip], r.discharge(20, 30)[:, ~skip]
    assert a.max() > 0 and np.array_equal(a, b)


@pytest.mark.parametrize("temp", [False, True])
def test_a_mask_set_in_mid_run(temp):
    got = []
    for flags in (True, False):
        m = _model(temp, flags)
        total = m.num_steps(ND)
        m.run_steps(DOY0, 0, ND, 0, 70)
        skip = _above(m.region, _cell_with_upstream(m.region))
        m.set_active_cells(~skip)
        m.run_steps(DOY0, 0, ND, 70, 80)
        m.set_active_cells(None)
        m.run_steps(DOY0, 0, ND, 80, total)
        got.append(_all(m, temp))
    _same(*got)


@pytest.mark.parametrize("mask,what", [(False, "upstream outflow"), (True, "grid barrier")])
def test_a_wait_that_runs_out_says_which(mask, what):
    from watergap2_gb300.gpu import WgError
    m = _model()
    if mask:
        m.set_active_cells(np.ones(m.region.ncell))
    m.barrier_test(1)
    m.run_steps(DOY0, 0, ND, 0, 10)
    with pytest.raises(WgError, match=what):
        m.synchronize()
