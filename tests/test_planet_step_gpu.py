"""One substep of free planets (AdvanceSystemRK5, src/Pframeforce.c:163-266,
with RungeKunta's Cash-Karp stages, src/RungeKunta.c:13-91) for one planet,
whose state the step keeps in registers, and for two, whose arrays it keeps in
shared memory, in a fixed and in a corotating frame, against numpy.

Tolerance: 2e-15 of the orbit's scale: a handful of roundings of 1.1e-16 in a
step whose displacement is 2e-3 of the radius (the fast build fuses
multiply-adds, so it rounds differently).
"""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 2e-15
A = [[], [1 / 5], [3 / 40, 9 / 40], [3 / 10, -9 / 10, 6 / 5], [-11 / 54, 5 / 2, -70 / 27, 35 / 27],
     [1631 / 55296, 175 / 512, 575 / 13824, 44275 / 110592, 253 / 4096]]
C = [37 / 378, 0.0, 250 / 621, 125 / 594, 0.0, 512 / 1771]


def _deriv(q, m):
    x, v = q[:2], q[2:]
    r3 = np.sum(x ** 2, axis=0) ** 1.5
    acc = -x / r3 - np.sum(m * x / r3, axis=1, keepdims=True)  # the star, and the indirect term
    return np.concatenate([v, acc])


def _step(q, m, dt):
    k = []
    for row in A:
        k.append(dt * _deriv(q + sum(a * s for a, s in zip(row, k)), m))
    return q + sum(c * s for c, s in zip(C, k))


@pytest.mark.parametrize("mode", ["parity", "fast"])
@pytest.mark.parametrize("planets,corot", [(1, 0), (1, 1), (2, 0)])
def test_free_planets_step(tmp_path, planets, corot, mode):
    import dustyfargoadsg_b200 as fb
    cfg = tmp_path / "p.cfg"
    cfg.write_text("# Planet Name   Distance   Mass    Accretion   Feels Disk   Feels Others\n" +
                   "".join("P%d  %g  1e-3  0.0  No  No\n" % (n, 1.0 + 0.5 * n) for n in range(planets)))
    p = fb.read_par(os.path.join(fb.CONFIG_DIR, "iso_128x384.par"), nrad=32, nsec=96, dt=2e-3, forced_circular=0,
                    corotating=corot, planetconfig=str(cfg))
    with fb.Disc(p, noise=1e-4, seed=3, mode=mode) as d:
        a = d.download()
        assert d.step().substeps == 1
        b = d.download()
    q = np.array([a["pl_" + k] for k in ("x", "y", "vx", "vy")])
    q = _step(q, a["pl_mass"], p.dt)
    if corot:  # OmegaFrame becomes the angle the planet turned through over dt; RotatePsys by it
        x0, y0 = a["pl_x"][0], a["pl_y"][0]
        ang = np.arcsin((x0 * q[1, 0] - q[0, 0] * y0) / (np.hypot(x0, y0) * np.hypot(q[0, 0], q[1, 0])))
        c, s = np.cos(ang), np.sin(ang)
        q = np.array([q[0] * c + q[1] * s, -q[0] * s + q[1] * c, q[2] * c + q[3] * s, -q[2] * s + q[3] * c])
    for n, k in enumerate(("x", "y", "vx", "vy")):
        assert np.max(np.abs(b["pl_" + k] - q[n])) <= TOL, (k, b["pl_" + k], q[n])
