"""Monthly grids of ensembles on both sides of the staging's thirty doubles per cell: put
into cell order on the device, or on the host where a row does not fit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_rows_that_do_not_fit_the_staging():
    from watergap2_gb300 import synthetic as sy
    from watergap2_gb300.gpu import Model
    region, nd = sy.region_small_swb(seed=5, ny=17, nx=31), 40
    P, T, S = sy.forcing(region, nd, seed=4, doy0=80)
    pf = np.random.default_rng(2).uniform(0.8, 1.2, 47)
    got = []
    for members in (30, 31, 47):
        m = Model(region, max_days=nd, precision="fp32", members=members, prec_factor=pf[:members])
        m.monthly_outputs(2, doy_day0=80)
        m.upload_forcing(0, P, T, S)
        m.run_days(80, 0, nd)
        got.append([np.asarray(m.monthly(k)).reshape(2, region.ncell, members)[:, :, :30]
                    for k in ("river_avail", "storage", "min_avail", "max_avail", "cell_runoff", "velocity")])
    assert got[0][0].max() > 0
    for other in got[1:]:
        for a, b in zip(got[0], other):
            assert np.array_equal(a, b)

