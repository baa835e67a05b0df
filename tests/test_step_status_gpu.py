"""What a DT reports about a state that goes bad between its substeps: the
substep's end tests it, on small grids in k_finish (one and two cells per
thread), on longer rings in k_cfl at the start of the next substep.

The failures are made on the host, by the ring profiles that the step itself
applies at every substep's end: the walls set the density of ring 1 to SigmaMed,
the damping towards the initial profiles pulls the energy to EnergyMed.  The
uploaded state is sound, so nothing is wrong at the first substep's start and
everything at the others'.
"""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRIDS = [(20, 384), (20, 1024), (20, 1025)]  # k_finish<1>, k_finish<2>, k_cfl
NAMES = (("SigmaMed", "sigma_med"), ("EnergyMed", "energy_med"), ("VthetaMed", "vtheta_med"),
         ("VradMed", "vrad_med"), ("GLOBAL_SoundSpeed", "global_soundspeed"))
RING = 1


def _adiabatic(nr, ns):
    """No viscosity: a ring without a sound speed would spread it.  The damping
    time is a hundredth of a substep or so: a damped ring takes its target."""
    import dustyfargoadsg_b200 as fb
    return fb.read_par(os.path.join(fb.CONFIG_DIR, "adiabatic_sg_512x1536.par"), nrad=nr, nsec=ns, self_gravity=0,
                       alphaviscosity=0.0, damp_to_axi=0, damp_to_ini=1, wkzrmin=0.5,
                       dampingtodynamicaltimeratio=1e-4)


def _isothermal(nr, ns):
    import dustyfargoadsg_b200 as fb
    return fb.read_par(os.path.join(fb.CONFIG_DIR, "iso_128x384.par"), nrad=nr, nsec=ns)


def _with_profile(disc, name, factor):
    """Uploads the disc's state with one ring of a profile times factor."""
    st = disc.download()
    st.update({k: disc.prof[a].copy() for k, a in NAMES})
    st[name][RING] *= factor
    disc.set_state(st)


@pytest.mark.parametrize("mode", ["parity", "fast"])
@pytest.mark.parametrize("nr,ns", GRIDS)
def test_nonfinite_after_a_substep_stops_the_dt(nr, ns, mode):
    import dustyfargoadsg_b200 as fb
    with fb.Disc(_isothermal(nr, ns), noise=1e-4, seed=2, mode=mode) as d:
        good = d.step()
        assert good.status == 0 and good.substeps >= 3
        _with_profile(d, "SigmaMed", np.nan)
        with pytest.raises(fb.FbError) as e:
            d.step()
        assert e.value.code == -5  # FB_ERR_NAN


@pytest.mark.parametrize("mode", ["parity", "fast"])
@pytest.mark.parametrize("nr,ns", GRIDS)
def test_negative_energy_after_a_substep_is_a_crash(nr, ns, mode):
    import dustyfargoadsg_b200 as fb
    from dustyfargoadsg_b200 import _ffi
    with fb.Disc(_adiabatic(nr, ns), noise=1e-4, seed=2, mode=mode) as d:
        _with_profile(d, "EnergyMed", -0.1)
        rep = d.step()
        assert rep.substeps >= 3
        assert rep.status == _ffi.FB_ERR_NEGATIVE
        assert rep.crashes == rep.crash_substeps == rep.substeps - 1
        assert rep.neg_density_substeps == 0
        crash = d.crash_state()
        assert 0.0 < crash["crash_time"] < d.p.dt
        neg = crash["energy"].reshape(nr, ns) < 0.0
        assert np.all(neg[RING]) and not np.any(np.delete(neg, RING, axis=0))


@pytest.mark.parametrize("mode", ["parity", "fast"])
@pytest.mark.parametrize("nr,ns", GRIDS)
def test_negative_density_after_a_substep_is_counted(nr, ns, mode):
    """Counted, but no crash: the energy test's result overwrites it."""
    import dustyfargoadsg_b200 as fb
    with fb.Disc(_adiabatic(nr, ns), noise=1e-4, seed=2, mode=mode) as d:
        _with_profile(d, "SigmaMed", -0.5)
        rep = d.step()
        assert rep.status == 0 and rep.crashes == 0 and rep.crash_substeps == 0
        assert rep.substeps >= 3 and rep.neg_density_substeps == rep.substeps - 1


@pytest.mark.parametrize("nr,ns", GRIDS)
def test_substep_cap(nr, ns, monkeypatch):
    import dustyfargoadsg_b200 as fb
    with fb.Disc(_isothermal(nr, ns), noise=1e-4, seed=2) as d:
        n = d.step().substeps
    for cap, ok in ((n, True), (n - 1, False)):
        monkeypatch.setenv("FB_MAX_SUBSTEPS", str(cap))  # read when the context is created
        with fb.Disc(_isothermal(nr, ns), noise=1e-4, seed=2) as d:
            if ok:
                assert d.step().substeps == n
            else:
                with pytest.raises(fb.FbError) as e:
                    d.step()
                assert e.value.code == -7  # FB_ERR_SUBSTEPS
