"""One or two DTs of small discs over the paths of the substep that the numpy
restatement of the step does not cover (self-gravity, particles, the other
edges, turbulent potential, rotating frames, free planets, radiative cooling,
damping towards the initial profiles, zeroed edge velocities), against states
recorded in golden/step_paths.npz by golden/make_step_paths.py.

The recording was made with the library of commit a5ab038, which runs every
step of the substep in a kernel of its own and whose step was compared with
the reference's own build.  Grids: 16 x 48 and 13 x 40 (tiles of k_sources cut in both
directions) and, for k_finish's two cells per thread, 8 x 400; discs with
self-gravity end their substeps in k_vr_damping, the other walled ones in
k_finish.

Tolerances, relative to each array's largest value (planets: distance): gas 1e-11, the parity bar
of a DT; particles 1e-10, their parity bar; the random stream and the numbers
of substeps and kicks exactly.
"""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
GOLDEN = os.path.join(HERE, "golden", "step_paths.npz")
TOL_GAS, TOL_DUST = 1e-11, 1e-10
GAS = ("dens", "vrad", "vtheta", "energy")

ISO, ADI, DUST = "iso_128x384.par", "adiabatic_sg_512x1536.par", "dust_256x768.par"
INI = dict(damp_to_axi=0, damp_to_ini=1, zero_vrad_bc=1)
OPEN = dict(wall_boundary=0, open_inner=1)
NONREF = dict(wall_boundary=0, non_reflecting=1)
GRAINS = dict(nbpart=300, sizeminpart=1e-6, sizemaxpart=1e-2, sizepartslope=3.5, rhopart=2.7, dustslope=0.0,
              rmindust=0.6, rmaxdust=1.8, dust_feel_turb=1, dust_feel_disk=1, dust_feel_planets=1)
BOULDERS = dict(GRAINS, sizeminpart=0.1, sizemaxpart=1.0, sizepartslope=1.0)
EXAMPLE = dict(rmin=0.4, rmax=2.5, wkzrmin=0.5, wkzrmax=2.1, beta_cooling=0, thermal_cooling=1)
LSA = dict(mhd_lsa=1, nbturbmodes=20, gammaturb=1e-3, high_m_cutoff=0, lsamodespeedup=1.0, turbrmin=0.5, turbrmax=2.0)

# name: (parameter file, rings, azimuths, DTs, overrides)
CASES = {
    "sg_adi": (ADI, 16, 48, 1, {}),
    "sg_adi_ini": (ADI, 16, 48, 1, INI),
    "sg_iso_ini": (ISO, 16, 48, 1, dict(INI, self_gravity=1, sgthicknesssmoothing=0.3)),
    "iso_ini": (ISO, 13, 40, 1, INI),
    "adi_ini": (ADI, 13, 40, 1, dict(INI, self_gravity=0)),
    "adi_ini_two_cells": (ADI, 8, 400, 1, dict(INI, self_gravity=0)),
    "adi_open": (ADI, 13, 40, 1, dict(OPEN, self_gravity=0)),
    "iso_open_kn": (ISO, 13, 40, 1, dict(OPEN, kn_open=1)),
    "iso_nonreflecting": (ISO, 13, 40, 1, NONREF),
    "cooling_nonreflecting_corot": (ADI, 13, 40, 1, dict(NONREF, self_gravity=0, corotating=1, forced_circular=0,
                                                         **EXAMPLE)),
    "iso_corot_free": (ISO, 13, 40, 1, dict(corotating=1, forced_circular=0)),
    "sg_adi_corot": (ADI, 16, 48, 1, dict(corotating=1)),
    "iso_lsa": (ISO, 13, 40, 1, LSA),
    "dust": (DUST, 13, 40, 2, GRAINS),
    "dust_boulders": (DUST, 13, 40, 2, dict(BOULDERS, dust_feel_turb=0)),
    "dust_adi": (ADI, 13, 40, 2, dict(BOULDERS, self_gravity=0)),
    "dust_sg_adi": (ADI, 16, 48, 2, dict(BOULDERS, dust_feel_sg=1)),
    "dust_sg_iso": (DUST, 16, 48, 1, dict(BOULDERS, self_gravity=1, sgthicknesssmoothing=0.3, dust_feel_sg=1)),
    # what a parameter file cannot ask for; overrides can
    "adi_implicit_odd": (ADI, 13, 41, 1, dict(self_gravity=0, radiative_diffusion=2)),
    "dust_lsa": (DUST, 13, 40, 2, dict(BOULDERS, **LSA)),
    "dust_corot": (DUST, 13, 40, 2, dict(BOULDERS, corotating=1)),
}


def run_case(fb, name, mode):
    """{array name: values} after the case's DTs."""
    par, nr, ns, dts, over = CASES[name]
    p = fb.read_par(os.path.join(fb.CONFIG_DIR, par), nrad=nr, nsec=ns, **over)
    with fb.Disc(p, noise=1e-3, seed=5, dust_seed=9 if p.nbpart else None, mode=mode) as d:
        sub = [d.step().substeps for _ in range(dts)]
        out = d.download()
        res = {k: out[k] for k in GAS + ("LostMass", "OmegaFrame", "pl_x", "pl_y")}
        res["substeps"] = np.array(sub)
        if p.nbpart:
            dust = d.dust()
            res.update({"pc_" + k: dust["pc_" + k] for k in d.DUST_ARRAYS})
            res["stream"] = np.array([dust["pc_rng_x"], dust["pc_kicks"]], dtype=np.uint64)
    return res


@pytest.mark.parametrize("mode", ["parity", "fast"])
@pytest.mark.parametrize("name", sorted(CASES))
def test_step_path_matches_recording(name, mode):
    import dustyfargoadsg_b200 as fb
    got = run_case(fb, name, mode)
    with np.load(GOLDEN) as z:
        want = {k.split("/", 1)[1]: z[k] for k in z.files if k.split("/", 1)[0] == name}
    assert set(got) == set(want)
    for k, w in want.items():
        g = np.asarray(got[k])
        if k in ("substeps", "stream"):
            np.testing.assert_array_equal(g, w, err_msg=k)
            continue
        # a planet's coordinates: of its distance (one of them is zero in the frame that follows it)
        scale = np.hypot(want["pl_x"], want["pl_y"]) if k in ("pl_x", "pl_y") else np.abs(w)
        err = np.max(np.abs(g - w)) / (np.max(scale) or 1.0)
        assert err <= (TOL_DUST if k.startswith("pc_") else TOL_GAS), (k, err)


@pytest.mark.parametrize("par", [ISO, ADI])
def test_damping_towards_the_initial_profiles(par):
    """The stage that the recorded discs' substeps end with, against numpy:
    EvanescentBoundary (src/SideEuler.c:796-950) with DampToIni and ZeroVradBC.
    Bar of the stages: 1e-12 of each field's largest value."""
    import dustyfargoadsg_b200 as fb
    from dustyfargoadsg_b200._ffi import FB_STAGE_DAMPING
    nr, ns, dt = 24, 72, 0.03
    p = fb.read_par(os.path.join(fb.CONFIG_DIR, par), nrad=nr, nsec=ns, self_gravity=0, rmin=0.4, rmax=2.5, wkzrmin=0.5,
                    wkzrmax=2.1, **INI)
    with fb.Disc(p, noise=1e-2, seed=4) as d:
        d.step()
        prof = {k: d.prof[k].copy() for k in ("sigma_med", "vtheta_med", "vrad_med", "energy_med")}
        f = {k: v.reshape(nr + 1, ns) for k, v in d.download().items() if k in GAS}
        d.stage(FB_STAGE_DAMPING, dt)
        got = d.download()
    radii = p.rmin * np.exp(np.arange(nr + 1) / nr * np.log(p.rmax / p.rmin))
    rmed = 2.0 / 3.0 * np.diff(radii ** 3) / np.diff(radii ** 2)
    zeroed = damped = 0
    for i in range(nr):
        lo, hi = rmed[i] < p.wkzrmin, rmed[i] > p.wkzrmax
        if not (lo or hi):
            continue
        damped += 1
        ref, end = (p.wkzrmin, rmed[0]) if lo else (p.wkzrmax, rmed[-1])
        lam = ((rmed[i] - ref) / (end - ref)) ** 2 * dt / (p.dampingtodynamicaltimeratio * rmed[i] ** 1.5)
        target = dict(dens=prof["sigma_med"][i], vtheta=prof["vtheta_med"][i], vrad=prof["vrad_med"][i],
                      energy=prof["energy_med"][i])
        zero = (lo and i <= 1) or (hi and i == nr - 1)
        zeroed += zero
        for k in GAS[:3] + ((GAS[3],) if p.energy_equation else ()):
            f[k][i] = (f[k][i] + lam * target[k]) / (1.0 + lam)
            if zero and k != "energy":
                f[k][i] = 0.0 if k == "vrad" else target[k]
    assert zeroed >= 2 and damped > zeroed
    for k in GAS:
        err = np.max(np.abs(got[k] - f[k].ravel())) / (np.max(np.abs(f[k])) or 1.0)
        assert err <= 1e-12, (k, err)
