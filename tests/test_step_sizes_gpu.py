"""The step on grids at the edges of its kernels' tiles: one DT of isothermal
and adiabatic discs (with and without viscous heating, both builds of the
library) against the plain numpy restatement of the step in perf/cases.py.

Sizes: rings and azimuths at, just below and just above whole tiles of
k_sources (27 azimuths, 11 or 27 rings), the smallest grids, grids narrower
than one tile, and both sides of k_finish's limits (one and two cells per
thread; rings longer than it takes).

Tolerance: the one-DT parity bar of this path, 1e-11 of each field's largest
value.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL_DT = 1e-11
SIZES = [(4, 16), (8, 26), (11, 27), (12, 28), (27, 53), (28, 54), (22, 81), (54, 55), (40, 200)]
BIG = [(110, 540), (109, 541), (20, 384), (20, 385), (20, 1024), (20, 1025), (300, 40)]
# (110, 540): two rings per warp of k_sources; (20, 1025), (300, 40): beyond k_finish


def _cases():
    for nr, ns in SIZES + BIG:
        yield dict(par="iso_128x384.par", nrad=nr, nsec=ns)
        yield dict(par="adiabatic_sg_512x1536.par", nrad=nr, nsec=ns, self_gravity=0)
    yield dict(par="adiabatic_sg_512x1536.par", nrad=28, nsec=80, self_gravity=0, viscous_heating=0)
    yield dict(par="adiabatic_sg_512x1536.par", nrad=28, nsec=80, self_gravity=0, beta_cooling=0)


@pytest.mark.parametrize("mode", ["parity", "fast"])
@pytest.mark.parametrize("case", list(_cases()), ids=lambda c: "%s_%dx%d%s" % (
    c["par"][:3], c["nrad"], c["nsec"], "_noheat" if c.get("viscous_heating") == 0 else
    "_nocool" if c.get("beta_cooling") == 0 else ""))
def test_one_dt_matches_numpy(case, mode):
    from perf import cases
    case = dict(case, kind="gas", mode=mode, dts=1)
    want = cases.exact(case, 17)
    state = cases.prepare(case, 17)
    got = cases.run(state)
    state["disc"].close()
    for k, x, y in zip(cases.FIELDS, got[1:5], want[1:5]):
        err = np.max(np.abs(x - y)) / (np.max(np.abs(y)) or 1.0)  # the isothermal energy is zero
        assert err <= TOL_DT, (k, err)
