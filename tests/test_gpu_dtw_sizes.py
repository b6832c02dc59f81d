"""The warping program at the sizes where its kernel changes form: traces that
end at, before and after a block of the traceback's rows, and candidate counts
with 32 .. 1 lanes per candidate, one and several candidates per lane, and few
rows of node costs at once. Shifts against the FP64 oracle (its decisions); over
many traces, with every number of lanes per candidate, equal to the bit."""
import multiprocessing
import os
from concurrent.futures import ProcessPoolExecutor

import numpy as np
import pytest

from oracle import oracle_dtw as D
from owl_b200 import _lib as L
from owl_b200.solver import MisfitOpts, dtw_time_shifts

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nt,m", [(3, 3), (32, 15), (33, 17), (34, 33), (65, 101), (96, 129), (97, 257), (129, 401),
                                  (40, 601), (33, 1101)])
def test_dtw_sizes(nt, m):
    rng = np.random.default_rng(nt + m)
    t = np.arange(nt)
    obs = np.stack([np.exp(-((t - nt * c) / (0.1 * nt)) ** 2) * np.cos(0.3 * t) for c in (0.4, 0.5, 0.6)])
    syn = np.stack([np.interp(t + s, t, o) for s, o in zip((0.7, -0.4, 1.3), obs)])
    obs, syn = ((a + 0.01 * rng.standard_normal(a.shape)).astype(np.float32) for a in (obs, syn))
    dt = 1e-3
    tlag = float(np.float32(0.5 * (m - 1) * dt))
    _, _, _, ref = D.adjoint_source([0, 3], syn, obs, None, dt=dt, tlag_max=tlag)
    tau = dtw_time_shifts(MisfitOpts(misfit=L.OWL_MISFIT_DTW, dt=dt, tlag_max=tlag), [0, 3], syn, obs)
    # the same decisions in the same double arithmetic, stored in single precision
    assert np.max(np.abs(tau - ref)) <= 1e-6, np.max(np.abs(tau - ref))


def _spread(ntr, nt, dt, seed):
    """gathers of five wavelets, the observed ones shifted slowly along the spread, and a little noise"""
    rng = np.random.default_rng(seed)
    t, span = np.arange(nt) * dt, (nt - 1) * dt
    f0 = 12.0 / span
    syn, obs = np.zeros((ntr, nt)), np.zeros((ntr, nt))
    for w in range(5):
        t0 = span * rng.uniform(0.15, 0.8) + np.linspace(0.0, 0.1 * span, ntr)
        a = rng.uniform(-1.0, 1.0, ntr) * 0.2 + rng.choice([-1.0, 1.0])
        lag = span * (0.02 * np.sin(np.linspace(0, 6, ntr) + w) + rng.uniform(-0.01, 0.01))
        for target, tc, amp in ((syn, t0, a), (obs, t0 + lag, a * rng.uniform(0.8, 1.2))):
            arg = (np.pi * f0 * (t[None, :] - tc[:, None])) ** 2
            target += amp[:, None] * (1.0 - 2.0 * arg) * np.exp(-arg)
    noise = 1e-3 * rng.standard_normal((2, ntr, nt))
    return (syn + noise[0]).astype(np.float32), (obs + noise[1]).astype(np.float32)


def _oracle_shifts(job):
    syn, obs, kw = job
    return D.adjoint_source([0, syn.shape[0]], syn, obs, None, **kw)[3]


@pytest.fixture(scope="module")
def pool():
    with ProcessPoolExecutor(min(16, os.cpu_count() or 1), mp_context=multiprocessing.get_context("spawn")) as p:
        yield p


# 32, 16, 8, 4, 2 lanes and one lane per candidate; the defaults on a long trace, and a distance without a cost of
# the shift itself (a negative weight), refined further, where neighbouring candidates come closest
CLOSE = dict(power=2.0, rcuml=-1.0, niter=12)


@pytest.mark.parametrize("nt,m,own", [(1001, 101, {}), (101, 9, {}), (41, 401, {}), (201, 9, CLOSE), (201, 31, CLOSE),
                                      (201, 63, CLOSE), (151, 101, CLOSE), (81, 201, CLOSE), (41, 401, CLOSE)])
def test_dtw_decisions_of_many_traces(pool, nt, m, own):
    dt, ntr = 1e-3, 128
    syn, obs = _spread(ntr, nt, dt, nt + m)
    tlag = float(np.float32(0.5 * (m - 1) * dt))
    kw = dict(dt=dt, tlag_max=tlag, **dict(own, rcuml=0.0) if own else {})
    ref = np.concatenate(list(pool.map(_oracle_shifts, [(syn[i:i + 8], obs[i:i + 8], kw) for i in range(0, ntr, 8)])))
    mo = MisfitOpts(misfit=L.OWL_MISFIT_DTW, dt=dt, tlag_max=tlag)
    if own:
        mo.dtw_loss_power, mo.dtw_rcuml, mo.dtw_niter = own["power"], own["rcuml"], own["niter"]
    tau = dtw_time_shifts(mo, [0, ntr], syn, obs)
    np.testing.assert_array_equal(tau, ref)


@pytest.mark.parametrize("m", [3857, 4095])
def test_dtw_most_candidates(m):
    """up to the documented limit of 4095 candidates"""
    dt, nt, niter = 1e-3, 9, 2
    syn, obs = _spread(1, nt, dt, m)
    tlag = float(np.float32(0.5 * (m - 1) * dt))
    ref = _oracle_shifts((syn, obs, dict(dt=dt, tlag_max=tlag, niter=niter)))
    tau = dtw_time_shifts(MisfitOpts(misfit=L.OWL_MISFIT_DTW, dt=dt, tlag_max=tlag, dtw_niter=niter), [0, 1], syn, obs)
    np.testing.assert_array_equal(tau, ref)
