"""The warping program at the sizes where its kernel changes form: traces that
end at, before and after a block of the traceback's rows, and candidate counts
with 32 .. 1 lanes per candidate, one and several candidates per lane, and few
rows of node costs at once. Shifts against the FP64 oracle (its decisions)."""
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
