"""Workspaces kept between the stateless calls (directions, gradient processing,
adjoint sources): calls of other kinds and sizes before, between and beside a call
do not change its bytes; a call that ends by an error leaves the next one alone;
idle workspaces do not change how a solver splits its shots."""
import ctypes as C
import os
import subprocess
import sys
import threading

import numpy as np
import pytest

from owl_b200 import _lib as L
from owl_b200.geometry import Receiver, Shot, Source
from owl_b200.optim import process, search_direction
from owl_b200.solver import MisfitOpts, RunOpts, SSGSolver, adjoint_source, dtw_time_shifts

HERE = os.path.dirname(os.path.abspath(__file__))
pytestmark = pytest.mark.gpu


def _rows(ntr, nt, seed):
    rng = np.random.default_rng(seed)
    t = np.arange(nt)
    obs = np.stack([np.exp(-((t - nt * c) / (0.08 * nt)) ** 2) * np.cos(0.25 * (t - nt * c))
                    for c in rng.uniform(0.3, 0.7, ntr)])
    syn = np.stack([np.interp(t + s, t, o) for s, o in zip(rng.uniform(-2, 2, ntr), obs)])
    return [(a + 0.01 * rng.standard_normal(a.shape)).astype(np.float32) for a in (syn, obs)]


def _adjoint(misfit, ntr, nt, **kw):
    syn, obs = _rows(ntr, nt, ntr + nt)
    return adjoint_source(MisfitOpts(misfit=misfit, dt=1e-3, **kw), [0, ntr // 2, ntr], syn, obs)


def _direction(n, nm):
    rng = np.random.default_rng(n)
    x = [rng.standard_normal(n).astype(np.float32) for _ in range(nm)]
    g = [(0.8 * a + 0.2 * rng.standard_normal(n)).astype(np.float32) for a in x]
    return [search_direction(m, x, g, x[0]) for m in (L.OWL_SEARCH_CG, L.OWL_SEARCH_LBFGS)]


def _smooth(shape, sigma):
    return [process(np.random.default_rng(3).standard_normal(shape).astype(np.float32), L.OWL_GRAD_SMOOTH, sigma)]


CALLS = {
    "envelope": lambda: _adjoint(L.OWL_MISFIT_ENVELOPE, 20, 301),
    "envelope short": lambda: _adjoint(L.OWL_MISFIT_ENVELOPE, 7, 64),
    "adaptive": lambda: _adjoint(L.OWL_MISFIT_ADAPTIVE, 12, 201, tlag_max=0.05),
    "waveform": lambda: _adjoint(L.OWL_MISFIT_WAVEFORM, 33, 500),
    "dtw": lambda: _adjoint(L.OWL_MISFIT_DTW, 9, 150, tlag_max=0.02),
    "dtw long": lambda: _adjoint(L.OWL_MISFIT_DTW, 4, 333, tlag_max=0.04),
    "direction": lambda: _direction(70001, 5),
    "direction small": lambda: _direction(300, 2),
    "smooth": lambda: _smooth((61, 83), [2.0, 3.0, 0.0]),
    "smooth wide": lambda: _smooth((400, 30), [95.0, 1.0, 0.0]),
}


def run_one(name, path):
    np.savez(path, *[np.asarray(a) for a in CALLS[name]()])


def _rejected():
    syn, obs = _rows(4, 100, 0)
    with pytest.raises(L.OwlError):
        adjoint_source(MisfitOpts(misfit=L.OWL_MISFIT_DTW, dt=1e-5, tlag_max=0.03), [0, 4], syn, obs)


def test_calls_do_not_see_each_other(tmp_path):
    """every call's outputs in any company equal those of a process of its own"""
    jobs = {}
    for i, name in enumerate(CALLS):
        out = str(tmp_path / f"{i}.npz")
        code = f"import sys; sys.path[:0] = [{os.path.dirname(HERE)!r}, {HERE!r}]; import test_gpu_workspaces as t; t.run_one({name!r}, {out!r})"
        jobs[name] = (subprocess.Popen([sys.executable, "-c", code]), out)
    ref = {}
    for name, (p, out) in jobs.items():
        assert p.wait(timeout=300) == 0, name
        ref[name] = list(np.load(out).values())
    bad = []

    def worker(seed):
        rng = np.random.default_rng(seed)
        for r in range(4):
            for name in rng.permutation(list(CALLS)):
                try:
                    got = CALLS[name]()
                    if any(not np.array_equal(np.asarray(a), b) for a, b in zip(got, ref[name])):
                        bad.append((seed, r, name))
                except Exception as e:  # noqa: BLE001
                    bad.append((seed, r, name, repr(e)))
            _rejected()

    threads = [threading.Thread(target=worker, args=(s,)) for s in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad


def test_error_leaves_the_next_call_alone():
    """A call on a kept workspace while another stream is being captured is refused, and the next call works."""
    import torch
    lib = L.load()
    n = 5000
    rng = np.random.default_rng(1)
    x = [torch.from_numpy(rng.standard_normal(n).astype(np.float32)).cuda() for _ in range(3)]
    g = [(0.7 * a).contiguous() for a in x]
    g[2] += 0.1
    out = torch.empty(n, device="cuda")
    ref = search_direction(L.OWL_SEARCH_LBFGS, x, g).clone()
    xs = (C.c_void_p * 3)(*[t.data_ptr() for t in x])
    gs = (C.c_void_p * 3)(*[t.data_ptr() for t in g])
    for _ in range(2):
        rc = L.OWL_OK
        graph = torch.cuda.CUDAGraph()
        with pytest.raises(Exception):
            with torch.cuda.graph(graph, stream=torch.cuda.Stream()):
                y = x[0] + 1
                rc = lib.owl_search_direction(L.OWL_SEARCH_LBFGS, n, 3, xs, gs, None, C.c_void_p(out.data_ptr()),
                                              L.OWL_MEM_DEVICE)
        assert rc == L.OWL_ERR_CUDA
        torch.cuda.synchronize()
        assert torch.equal(search_direction(L.OWL_SEARCH_LBFGS, x, g), ref)
    del y


def test_idle_workspaces_do_not_change_the_batches():
    import torch
    nx, nz, nshots = 900, 900, 96
    vp = np.full((nz, nx), 2000.0, dtype=np.float32)
    shots = [Shot(k + 1, [Source(x=300.0 + 100.0 * k, z=500.0, f0=12.0)], [Receiver(x=1000.0, z=1000.0)])
             for k in range(nshots)]

    def solver():
        s = SSGSolver(L.OWL_ACOUSTIC_ISO_2D, nx, nz, 10.0, 10.0, 1e-3, 6, pml=10, f0_max=12.0, max_shots=nshots)
        s.set_model(vp, vp)
        return s, s.prepare(shots)

    syn, obs = _rows(592, 1001, 5)
    mo = MisfitOpts(misfit=L.OWL_MISFIT_DTW, dt=1e-3, tlag_max=0.08)  # back-pointers of about 200 MB
    warm = dtw_time_shifts(mo, [0, 592], syn, obs)
    s, ps = solver()
    s.forward(ps, RunOpts(shots_per_launch=1))
    del s
    torch.cuda.empty_cache()
    fill = torch.empty(torch.cuda.mem_get_info()[0] - (1400 << 20), dtype=torch.uint8, device="cuda")
    s, ps = solver()
    with pytest.raises(L.OwlError) as e:  # 96 shots at once do not fit: the idle workspaces go
        s.forward(ps, RunOpts(shots_per_launch=nshots))
    assert e.value.code == L.OWL_ERR_OOM
    del s
    s, ps = solver()
    a = s.forward(ps, RunOpts())
    alone = s.last_info.shots_per_launch
    del s
    np.testing.assert_array_equal(dtw_time_shifts(mo, [0, 592], syn, obs), warm)
    s, ps = solver()
    b = s.forward(ps, RunOpts())
    # (a shot takes 25 MB: the workspace held back would cost about eight)
    assert 8 <= alone < nshots and abs(s.last_info.shots_per_launch - alone) <= 1
    np.testing.assert_array_equal(a, b)
    del fill
