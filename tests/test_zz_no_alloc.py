"""GPU test of fb_transport_noalloc, the allocation-free transport entry point.

It exists for host codes that cannot call cudaMalloc: the step embedded in a
GPU application that owns the device-memory budget, or called from a region
where an allocation (which may synchronize the device) is not acceptable.
Its scratch is a fixed file-scope device array shared by all calls, so the
test makes two calls in a row (the second one sees the first one's leftover
scratch) on each of two grids, and checks every result, and the ring-0
outflow it reports, against the allocating path through a context,
fb_stage(ctx, FB_STAGE_TRANSPORT, dt), within the stage tolerance the other
GPU tests use.  Only the first call on a device may make the driver allocate
(it loads the kernels); the test checks that the device's free memory is the
same before and after every later call.
"""
import ctypes as C
import os

import numpy as np
import pytest

from tests import _oracle

pytestmark = pytest.mark.gpu

TOL_STAGE = 1e-12
FIELDS = ("dens", "vrad", "vtheta", "energy")
_setup_done = [False]  # the first call of this process on the device has been made


def _run_pair(par, dt):
    import torch

    import dustyfargoadsg_b200 as fb
    from dustyfargoadsg_b200 import _ffi
    lib = _ffi.load()
    p = fb.read_par(par)
    with fb.Disc(p, noise=1e-4, seed=11) as disc:
        start = disc.download()
        disc.stage(_ffi.FB_STAGE_TRANSPORT, dt)
        ref1 = disc.download()
        disc.stage(_ffi.FB_STAGE_TRANSPORT, dt)
        ref2 = disc.download()
    torch.cuda.synchronize()
    t = {k: torch.tensor(start[k], dtype=torch.float64, device="cuda") for k in FIELDS}
    ptr = {k: C.c_void_p(t[k].data_ptr()) for k in FIELDS}
    prev_lost = start["LostMass"]
    for ref in (ref1, ref2):
        torch.cuda.synchronize()
        free0 = torch.cuda.mem_get_info()[0]
        lost = C.c_double(0.0)
        rc = lib.fb_transport_noalloc(C.byref(p), ptr["dens"], ptr["vrad"], ptr["vtheta"], ptr["energy"],
                                      dt, None, C.byref(lost))
        assert rc == 0, lib.fb_noalloc_last_error().decode()
        torch.cuda.synchronize()
        if _setup_done[0]:
            assert torch.cuda.mem_get_info()[0] == free0, "a call after the first one allocated device memory"
        _setup_done[0] = True
        for k in FIELDS:
            got = t[k].cpu().numpy()
            err = _oracle.rel_err(got, ref[k])
            assert err <= TOL_STAGE, (k, err)
        # the ring-0 outflow of this call, as the context accumulates it
        want = ref["LostMass"] - prev_lost
        prev_lost = ref["LostMass"]
        assert abs(lost.value - want) <= TOL_STAGE * max(abs(want), abs(ref["LostMass"])), (lost.value, want)


def test_transport_noalloc_matches_context_path(tmp_path):
    iso = os.path.join(_oracle.CONFIG_DIR, "iso_128x384.par")
    adi = os.path.join(_oracle.CONFIG_DIR, "adiabatic_sg_512x1536.par")
    _run_pair(_oracle.write_par(iso, str(tmp_path), Nrad=48, Nsec=144), 0.02)
    d2 = tmp_path / "adi"
    d2.mkdir()
    _run_pair(_oracle.write_par(adi, str(d2), Nrad=64, Nsec=192, SelfGravity="No"), 0.005)


def test_transport_noalloc_refuses_oversized_grid(tmp_path):
    import dustyfargoadsg_b200 as fb
    from dustyfargoadsg_b200 import _ffi
    lib = _ffi.load()
    p = fb.read_par(os.path.join(_oracle.CONFIG_DIR, "adiabatic_sg_512x1536.par"))
    dummy = C.c_void_p(16)  # never dereferenced: the size check comes first
    rc = lib.fb_transport_noalloc(C.byref(p), dummy, dummy, dummy, dummy, 0.01, None, None)
    assert rc == -1
    assert b"too large" in lib.fb_noalloc_last_error()


def _call(lib, p, t, dt, stream=None, lost=None):
    ptr = [C.c_void_p(t[q].data_ptr()) for q in range(4)]
    return lib.fb_transport_noalloc(C.byref(p), *ptr, dt, C.c_void_p(stream),
                                    C.byref(lost) if lost is not None else None)


def test_calls_in_a_row_reuse_the_host_table(tmp_path):
    """Back-to-back calls on one stream, grids and calls with and without
    lost_mass alternating: a call must not see the tables of the next one, and
    each gives what a call on its own gives, to the last bit."""
    import torch

    import dustyfargoadsg_b200 as fb
    lib = fb.load()
    adi = os.path.join(_oracle.CONFIG_DIR, "adiabatic_sg_512x1536.par")
    runs = []
    for nr, ns, dt in ((48, 144, 0.02), (130, 390, 0.004), (17, 61, 0.03)):
        p = fb.read_par(adi, nrad=nr, nsec=ns, self_gravity=0)
        with fb.Disc(p, noise=1e-2, seed=nr) as disc:
            s = disc.download()
        start = torch.tensor(np.stack([s[k] for k in FIELDS]), device="cuda")
        alone, lost = start.clone(), C.c_double()
        torch.cuda.synchronize()
        assert _call(lib, p, alone, dt, lost=lost) == 0
        torch.cuda.synchronize()
        runs.append((p, dt, start, alone, lost.value))
    outs = []
    work = [(n, bool(with_lost), runs[n][2].clone()) for n, with_lost in
            ((0, 0), (1, 0), (2, 1), (1, 1), (0, 0), (2, 0), (0, 1), (1, 0), (2, 0))]
    torch.cuda.synchronize()
    for n, with_lost, t in work:
        lost = C.c_double() if with_lost else None
        assert _call(lib, runs[n][0], t, runs[n][1], lost=lost) == 0
        outs.append(lost.value if with_lost else None)
    torch.cuda.synchronize()
    for (n, _, t), lost in zip(work, outs):
        assert torch.equal(t, runs[n][3])
        assert lost is None or lost == runs[n][4]


def test_call_on_a_capturing_stream_is_refused(tmp_path):
    """With an error, leaving the capture valid; the next call works."""
    import torch

    import dustyfargoadsg_b200 as fb
    lib = fb.load()
    p = fb.read_par(os.path.join(_oracle.CONFIG_DIR, "iso_128x384.par"), nrad=32, nsec=96)
    with fb.Disc(p, noise=1e-4, seed=1) as disc:
        s = disc.download()
    start = torch.tensor(np.stack([s[k] for k in FIELDS]), device="cuda")
    t, x, lost = start.clone(), torch.zeros(8, device="cuda"), C.c_double()
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    for given in (lost, None):
        with torch.cuda.graph(graph, stream=stream):
            x.add_(1.0)
            rc = _call(lib, p, t, 0.01, stream=stream.cuda_stream, lost=given)
        assert rc == -3 and b"capturing" in lib.fb_noalloc_last_error()  # FB_ERR_CUDA
        graph.replay()
        torch.cuda.synchronize()
        graph.reset()
    assert float(x.sum()) == 16.0 and torch.equal(t, start)
    assert _call(lib, p, t, 0.01, lost=lost) == 0
    torch.cuda.synchronize()
    assert not torch.equal(t, start) and bool(torch.isfinite(t).all())
