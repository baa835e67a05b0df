"""The implicit radiative diffusion's solver on both sides of its size limits
(one to three cells per colour and thread of the cluster, grids the cluster
does not hold, ring counts that leave CTAs short or empty), against a plain
numpy restatement of the red-black iteration (SORsolver_RadiativeDiffusion,
src/SourceEuler.c:1878-2052) with a constant opacity.

A disc advances one substep of dt = DT with the diffusion on; the same disc
without it starts from the energy numpy solves for.  Both take the same gas
step, so the states must agree to its rounding.

Tolerance: the one-DT parity bar of this path, 1e-11 of each field's largest
value; the diffusion must change the energy by far more.
"""
import math
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL_DT = 1e-11
SIZES = [(4, 16), (12, 26), (18, 64), (19, 64), (35, 400), (66, 256), (67, 258), (128, 384), (132, 400)]


def _lambda(R):
    return np.where(R <= 2.0, 2.0 / (3.0 + np.sqrt(9.0 + 10.0 * R * R)),
                    10.0 / (10.0 * R + 9.0 + np.sqrt(180.0 * R + 81.0)))


def _solve(p, e, rho, dt):
    """Energy after the implicit diffusion of one substep."""
    from perf.cases import _Grid
    g, nr, ns = _Grid(p), p.nrad, p.nsec
    ul, um = 1.49598e11, 1.9891e30
    ut, uT = math.sqrt(ul ** 3 / 6.673e-11 / um), 2.35 * 8.0841643e-15 * um / ul
    sigma = 5.6704e-8 / um * ut ** 3 * uT ** 4
    opacity = p.imposedconstantopacity * 0.1 * ul ** -2.0 * um
    gam, c = p.adiabaticindex, lambda a: np.asarray(a)[:, None]
    t = (gam - 1.0) * e / rho
    a = c(g.idrm[1:]) * (t[1:] - t[:-1])
    b = c(1.0 / g.rmed[:-1]) / g.dphi * (np.roll(t, -1, 1) - t)[:-1]
    tt, rr, rm = t[:-1], rho[:-1], c(g.rmed[:-1])
    R = 8.0 * np.sqrt(gam * tt) * rm ** 1.5 / rr / opacity * (np.hypot(a, b) / tt)
    chi = 64.0 * sigma * _lambda(R) * gam * (gam - 1.0) * tt ** 4 * rm ** 3 / rr ** 2 / opacity
    chi = np.concatenate([chi, chi[-1:]])
    i = slice(1, nr - 1)
    rm, rs, ri = c(g.rmed), c(g.rsup), c(g.rinf)
    up = ((rm[2:] - rs[i]) * chi[i] + (rs[i] - rm[i]) * chi[2:]) / (rm[2:] - rm[i])
    lo = ((rm[i] - ri[i]) * chi[:-2] + (ri[i] - rm[:-2]) * chi[i]) / (rm[i] - rm[:-2])
    ids = 1.0 / (rs - ri)[i]
    A = -dt * rs[i] * ids * up / rm[i] / (rm[2:] - rm[i])
    B = -dt * ri[i] * ids * lo / rm[i] / (rm[i] - rm[:-2])
    C = -dt * 0.5 * (chi + np.roll(chi, -1, 1))[i] / rm[i] ** 2 / g.dphi ** 2
    D = -dt * 0.5 * (chi + np.roll(chi, 1, 1))[i] / rm[i] ** 2 / g.dphi ** 2
    E, F = 1.0 - A - B - C - D, t[i].copy()

    def resid():
        return A * t[2:] + B * t[:-2] + C * np.roll(t, -1, 1)[i] + D * np.roll(t, 1, 1)[i] + E * t[i] - F

    init = np.abs(resid()).sum()
    odd = ((np.arange(1, nr - 1)[:, None] + np.arange(ns)[None, :]) & 1) == 1
    for _ in range(100000):
        norm = 0.0
        for cells in (odd, ~odd):
            r = resid()
            norm += np.abs(r[cells]).sum()
            t[i] = np.where(cells, t[i] - 1.97 * r / E, t[i])
        if norm < 1e-4 * init:
            break
    return rho * t / (gam - 1.0)


@pytest.mark.parametrize("mode", ["parity", "fast"])
@pytest.mark.parametrize("nr,ns", SIZES)
def test_solver_matches_numpy(nr, ns, mode):
    import dustyfargoadsg_b200 as fb
    over = dict(nrad=nr, nsec=ns, self_gravity=0, dt=2e-4, constant_opacity=1, imposedconstantopacity=1e-3)
    path = os.path.join(fb.CONFIG_DIR, "adiabatic_sg_512x1536.par")
    with fb.Disc(fb.read_par(path, radiative_diffusion=2, **over), noise=1e-2, seed=9, mode=mode) as d:
        start = d.download()
        rep = d.step()
        got = d.download()
        prof = {k: d.prof[v].copy() for k, v in (("SigmaMed", "sigma_med"), ("EnergyMed", "energy_med"),
                                                 ("VthetaMed", "vtheta_med"), ("VradMed", "vrad_med"),
                                                 ("GLOBAL_SoundSpeed", "global_soundspeed"))}
    assert rep.substeps == 1
    p = fb.read_par(path, **over)
    e, rho = (start[k].reshape(nr + 1, ns)[:nr] for k in ("energy", "dens"))
    solved = _solve(p, e, rho, p.dt)
    assert np.max(np.abs(solved - e) / e) > 100 * TOL_DT  # the coarsest grids diffuse by 2e-8 in so short a DT
    state = dict(start, **prof)
    state["energy"] = np.concatenate([solved.ravel(), start["energy"][nr * ns:]])
    with fb.Disc(p, state=state, mode=mode) as d:
        assert d.step().substeps == 1
        want = d.download()
    for k in ("dens", "vrad", "vtheta", "energy"):
        err = np.max(np.abs(got[k] - want[k])) / np.max(np.abs(want[k]))
        assert err <= TOL_DT, (k, err)
