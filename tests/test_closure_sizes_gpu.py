"""The closure's convolution and weight-gradient kernels where the walks over
the rings can go wrong: the smallest grid, a ring count that no walk divides,
a last walk shorter than the others, and more samples than one wave of CTAs
holds, against the float64 restatement (which rounds to bfloat16 where the GPU
stores bfloat16).

Tolerances are those of the tests at 8x64 cells: an FP32 sum next to a
rounding boundary may round an activation to the other bfloat16, one part in
256 of that value, and such flips are independent of one another.
"""
import ctypes as C
import os

import numpy as np
import pytest

from tests import _oracle
from tests import closure_ref as R
from tests.test_closure_gpu import _closure, _dp, _fp, _geometry

pytestmark = pytest.mark.gpu
ISO = os.path.join(_oracle.CONFIG_DIR, "iso_128x384.par")


@pytest.mark.parametrize("nr,ns,batch", [(4, 64, 1), (41, 192, 1), (67, 128, 3), (4, 64, 300)])
def test_loss_and_gradients(tmp_path, nr, ns, batch):
    from dustyfargoadsg_b200 import Disc, _ffi, read_par
    p = read_par(_oracle.write_par(ISO, str(tmp_path), Nrad=nr, Nsec=ns))
    _, surf, _ = _geometry(p)
    params = R.init_params(seed=nr, scale=0.6)
    rng = np.random.RandomState(ns)
    x = R.bf16_round(rng.uniform(-1, 1, (batch, nr, ns, 16)))
    y = rng.standard_normal((batch, nr, ns)) * 0.05
    sig = rng.uniform(0.5, 2.0, (batch, nr)).astype(np.float32).astype(np.float64)
    scale, w = 0.02, 1.5
    with Disc(p) as disc:
        lib = disc.lib
        c = _closure(disc, batch, batch)
        try:
            wt, bt = R.flatten(params)
            _ffi.check(lib.fb_closure_params(c, _fp(wt), _fp(bt), 0), "params")
            _ffi.check(lib.fb_closure_scales(c, _dp(np.array([scale, 1.0, 1.0])), _dp(np.array([w, 1.0, 1.0])), 0),
                       "scales")
            for s in range(batch):
                ys = np.zeros((3, nr, ns), dtype=np.float32)
                ys[0] = y[s]
                _ffi.check(lib.fb_closure_set_sample(c, s, _fp(np.ascontiguousarray(x[s], dtype=np.float32)), _fp(ys),
                                                     _fp(np.ascontiguousarray(sig[s], dtype=np.float32))), "sample")
            out = np.zeros(nr * ns * 16, dtype=np.float32)
            _ffi.check(lib.fb_closure_infer(c, None, batch - 1, _fp(out)), "infer")
            gw, gb, loss = np.zeros_like(wt), np.zeros_like(bt), C.c_double()
            _ffi.check(lib.fb_closure_loss_grad(c, 0, batch, C.byref(loss), _fp(gw), _fp(gb)), "loss_grad")
        finally:
            lib.fb_closure_destroy(c)
    ref = R.forward(params, x[-1:], bf16=True)[0].ravel()
    assert np.linalg.norm(out - ref) <= 2e-3 * np.linalg.norm(ref)
    want, grads = R.loss_and_grads(params, x, y, scale, w, surf, sig, bf16=True)
    assert abs(loss.value - want) <= 1e-3 * want
    rw, rb = R.flatten([(g[0], g[1]) for g in grads])
    ow = ob = 0
    for cin, cout in R.LAYERS:
        n = cout * 9 * cin
        for got, ref, at, size in ((gw, rw, ow, n), (gb, rb, ob, cout)):
            assert np.linalg.norm((got - ref)[at:at + size]) <= 1e-2 * np.linalg.norm(ref[at:at + size])
        ow, ob = ow + n, ob + cout


def test_gradients_without_a_loss(tmp_path):
    """The loss is optional: without it the gradients are the same ones.
    Tolerance: two runs add the CTAs' FP32 sums in another order, at most some
    300 partial sums of 6e-8 each; 1e-5 of the norm."""
    from dustyfargoadsg_b200 import Disc, _ffi, read_par
    nr, ns, batch = 96, 256, 8
    params = R.init_params(seed=3, scale=0.6)
    rng = np.random.RandomState(1)
    with Disc(read_par(_oracle.write_par(ISO, str(tmp_path), Nrad=nr, Nsec=ns))) as disc:
        lib = disc.lib
        c = _closure(disc, batch, batch)
        try:
            wt, bt = R.flatten(params)
            _ffi.check(lib.fb_closure_params(c, _fp(wt), _fp(bt), 0), "params")
            _ffi.check(lib.fb_closure_scales(c, _dp(np.array([0.02, 1.0, 1.0])), _dp(np.array([1.5, 1.0, 1.0])), 0),
                       "scales")
            for s in range(batch):
                x, y = rng.uniform(-1, 1, (nr, ns, 16)), rng.standard_normal((3, nr, ns)) * 0.05
                _ffi.check(lib.fb_closure_set_sample(c, s, _fp(x.astype(np.float32)), _fp(y.astype(np.float32)),
                                                     _fp(np.ones(nr, dtype=np.float32))), "sample")
            runs = []
            for loss in (C.byref(C.c_double()), None, None, None):
                gw, gb = np.zeros_like(wt), np.zeros_like(bt)
                _ffi.check(lib.fb_closure_loss_grad(c, 0, batch, loss, _fp(gw), _fp(gb)), "loss_grad")
                runs.append((gw, gb))
        finally:
            lib.fb_closure_destroy(c)
    for got in runs[1:]:
        for g, w in zip(got, runs[0]):
            assert np.linalg.norm(w) > 0.0 and np.linalg.norm(g - w) <= 1e-5 * np.linalg.norm(w)
