"""Search directions and smoothing at the sizes where their launches change
form: one block, a ragged last block, more cells than the grid's threads; one
pair (the oldest is the newest) up to ten; filters whose weights travel in the
launch parameters and longer ones; one, two and three smoothed axes."""
import numpy as np
import pytest

import oracle.oracle_optim as O
from owl_b200 import _lib as L
from owl_b200.optim import process, search_direction

from cases import rel
from test_gpu_optim import _history

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 255, 257, 2 * 148 * 256 + 1])
@pytest.mark.parametrize("nm", [2, 3, 11])
@pytest.mark.parametrize("method", [L.OWL_SEARCH_CG, L.OWL_SEARCH_LBFGS])
def test_search_direction_sizes(n, nm, method):
    x, g = _history(n, nm, seed=n + nm)
    prev = np.random.default_rng(5).standard_normal(n).astype(np.float32)
    ref = O.search_direction(method, x, g, prev)
    got = search_direction(method, x, g, prev)
    # float32 storage of the direction between the pairs' updates
    assert rel(got, ref) < 1e-5, rel(got, ref)


def test_zero_curvature_pairs_drop_out():
    x, g = _history(1000, 4)
    x[2], g[2] = x[1].copy(), g[1].copy()  # s = y = 0
    ref = O.search_direction(L.OWL_SEARCH_LBFGS, x, g, None)
    assert rel(search_direction(L.OWL_SEARCH_LBFGS, x, g), ref) < 1e-5


@pytest.mark.parametrize("shape,sigma", [((40, 57), (2.0, 0.0, 0.0)), ((40, 57), (0.0, 3.3, 0.0)), ((301, 20), (85.3, 1.0, 0.0)),
                                         ((301, 9), (90.0, 0.4, 0.0)), ((13, 11, 17), (1.5, 2.0, 6.0))])
def test_smoothing_forms(shape, sigma):
    f = np.random.default_rng(4).standard_normal(shape).astype(np.float32)
    ref = np.asarray(f, dtype=np.float64)
    # the axes as the library orders them: z, then x (2D) or y, x (3D)
    for ax, sg in enumerate(sigma[: len(shape)]):
        if sg == 0:
            continue
        rad = max(1, int(np.ceil(3 * np.float32(sg))))
        w = np.exp(-0.5 * np.arange(-rad, rad + 1.0) ** 2 / float(np.float32(sg)) ** 2)
        w /= w.sum()
        p = np.pad(ref, [(rad, rad) if a == ax else (0, 0) for a in range(len(shape))], mode="edge")
        ref = sum(w[k] * np.take(p, range(k, k + shape[ax]), axis=ax) for k in range(2 * rad + 1))
    got = process(f, L.OWL_GRAD_SMOOTH, list(sigma))
    assert rel(got, ref) < 2e-6, rel(got, ref)


@pytest.mark.parametrize("n", [4 * 148 * 256 - 1, 4 * 148 * 256 + 1, 4 * 4 * 148 * 256 + 300])
@pytest.mark.parametrize("nm", [2, 4])
def test_several_cells_per_thread(n, nm):
    """one cell less and more than the grid's threads, and more than they take in one round"""
    x, g = _history(n, nm, seed=n + nm)
    ref = O.search_direction(L.OWL_SEARCH_LBFGS, x, g, None)
    assert rel(search_direction(L.OWL_SEARCH_LBFGS, x, g), ref) < 1e-5
