"""2D acoustic segments with the state resident in shared memory against the
step-by-step launches: the traces equal to the bit, gradients to FP32 rounding,
at the sizes where the split over a cluster's CTAs and the four-cell groups can
go wrong (ragged rows, one and many CTAs, rows of x-PML groups that meet)."""
import numpy as np
import pytest

from owl_b200 import _lib as L
from owl_b200.geometry import Receiver, Shot, Source
from owl_b200.solver import RunOpts, SSGSolver

pytestmark = pytest.mark.gpu

# one launch per kernel and step, one cell per thread (the four-cell kernels round a few sums differently)
STEPWISE = RunOpts(use_graph=-1, checkpoint_interval=25, tile_z=8, shots_per_cta=1)


def model(nz, nx, seed=3):
    rng = np.random.default_rng(seed)
    vp = (1800 + 900 * np.linspace(0, 1, nz)[:, None] + 200 * rng.random((nz, nx))).astype(np.float32)
    return vp, (310 * vp ** 0.25).astype(np.float32)


def shots_of(nshots, nx, nz, fs, nrec=None, mechanism="explosion"):
    out = []
    for k in range(nshots):
        srcs = [Source(x=10.0 * nx * (0.2 + 0.6 * k / max(1, nshots - 1)) + 3.3, z=31.7, f0=12.0, mechanism=mechanism),
                Source(x=10.0 * nx * 0.5, z=10.0 * (nz - 4), f0=9.0, amp=0.7, t0=0.02, mechanism=mechanism)]
        # on and off the nodes, near the surface, down a column that crosses every CTA, one switched off
        recs = [Receiver(x=20.0 + 17.3 * i, z=20.0) for i in range(min(nx // 2, nrec or nx))]
        recs += [Receiver(x=5.0 * nx + 1.0, z=0.0 if k % 2 else 7.0 + 10.0 * j) for j in range(0, nz - 2, 3)]
        recs += [Receiver(x=40.0, z=40.0, weight=0.0), Receiver(x=30.0, z=1.5 if fs else 15.0)]
        if nrec:
            recs = (recs * (nrec // len(recs) + 1))[:nrec]
        out.append(Shot(k + 1, srcs[: 1 + k % 2], recs))
    return out


CASES = [
    # nx, nz, pml, half, fs, shots, nt
    (40, 30, 8, 4, False, 1, 140),    # smallest: few rows per CTA
    (61, 47, 10, 4, True, 3, 130),    # odd sizes, free surface
    (64, 48, 10, 8, False, 2, 120),   # 16th order
    (77, 53, 11, 8, True, 2, 120),    # 16th order, free surface, ragged last group
    (131, 203, 20, 4, False, 5, 90),  # more rows than columns, z-PML rows in several CTAs
    (401, 201, 20, 4, False, 20, 60), # the benchmark grid, more shots than clusters
    (9, 120, 5, 4, True, 2, 100),     # x-PML groups that meet, narrow rows
    (250, 9, 3, 4, False, 2, 100),    # few rows
]


@pytest.mark.parametrize("nx,nz,pml,half,fs,nshots,nt", CASES)
def test_resident_segments_equal_step_launches(nx, nz, pml, half, fs, nshots, nt):
    vp, rho = model(nz, nx)
    s = SSGSolver(L.OWL_ACOUSTIC_ISO_2D, nx, nz, 10.0, 10.0, 1e-3, nt, pml=pml, fdhalf=half, free_surface=fs,
                  f0_max=12.0, max_shots=nshots)
    s.set_model(vp, rho)
    ps = s.prepare(shots_of(nshots, nx, nz, fs))
    a = s.forward(ps, RunOpts())
    launches = s.last_info.gpu_launches
    b = s.forward(ps, STEPWISE)
    assert launches < nt and s.last_info.gpu_launches > 2 * nt  # one launch against step by step
    assert np.all(np.isfinite(b)) and np.abs(b).max() > 0
    np.testing.assert_array_equal(a, b)
    obs = (0.5 * b).astype(np.float32)
    syn = [np.zeros_like(b) for _ in range(2)]
    m0, g0 = s.gradient(ps, obs, opts=RunOpts(checkpoint_interval=25), seis_out=syn[0])
    m1, g1 = s.gradient(ps, obs, opts=STEPWISE, seis_out=syn[1])
    np.testing.assert_array_equal(syn[0], syn[1])
    np.testing.assert_array_equal(m0, m1)
    for p in range(2):
        h0, h1 = np.split(g0, 2)[p], np.split(g1, 2)[p]
        # sums over the steps in another order: a few FP32 roundings of the largest terms
        assert np.linalg.norm(h0 - h1) <= 2e-6 * np.linalg.norm(h1)


def close(a, b):
    """The automatic step kernels may be the four-cell ones, which round a few sums differently."""
    assert np.linalg.norm(a - b) <= 2e-6 * np.linalg.norm(b)


def test_what_stays_step_by_step():
    """Force sources, more traces than a CTA's threads hold, taps beyond the updated nodes, explicit tiles and
    plain launches."""
    nx, nz, nt = 64, 48, 60
    vp, rho = model(nz, nx)
    s = SSGSolver(L.OWL_ACOUSTIC_ISO_2D, nx, nz, 10.0, 10.0, 1e-3, nt, pml=10, f0_max=12.0, max_shots=2)
    s.set_model(vp, rho)
    for shots in (shots_of(2, nx, nz, False, mechanism="force"), shots_of(1, nx, nz, False, nrec=1500)):
        ps = s.prepare(shots)
        a = s.forward(ps, RunOpts())
        assert s.last_info.gpu_launches > 2 * nt
        close(a, s.forward(ps, STEPWISE))
    # taps beyond the absorbing layer of a narrow one, where no node is updated
    narrow = SSGSolver(L.OWL_ACOUSTIC_ISO_2D, nx, nz, 10.0, 10.0, 1e-3, nt, pml=2, f0_max=12.0)
    narrow.set_model(vp, rho)
    ps = narrow.prepare([Shot(1, [Source(x=1.3, z=2.7, f0=12.0)], [Receiver(x=2.0 + 9.0 * i, z=4.0) for i in range(20)])])
    a = narrow.forward(ps, RunOpts())
    assert narrow.last_info.gpu_launches > 2 * nt
    close(a, narrow.forward(ps, STEPWISE))
    ps = s.prepare(shots_of(2, nx, nz, False))
    a = s.forward(ps, RunOpts())
    assert s.last_info.gpu_launches < nt
    for o in (RunOpts(tile_z=4, shots_per_cta=1), RunOpts(tile_z=8), STEPWISE):
        b = s.forward(ps, o)
        assert s.last_info.gpu_launches > 2 * nt
        np.testing.assert_array_equal(a, b)


def spread(nx, nz, half, pml, fs, pattern):
    """Receivers off the nodes: on every row, above a free surface, beside the sources, out to the edges of the
    absorbing layer; `pattern` picks nodes along x, along z, both or none."""
    ox, oz = {"x": (0.0, 3.7), "z": (4.1, 0.0), "both": (0.0, 0.0), "none": (4.1, 3.7)}[pattern]
    lo, hi = -10.0 * min(pml - 1, 3), 10.0 * min(pml - 1, 3)
    recs = [Receiver(x=10.0 * (nx // 3) + ox, z=10.0 * k + oz, weight=1.0 - 0.01 * (k % 5)) for k in range(nz - 1)]
    recs += [Receiver(x=lo + ox + (10.0 * nx + hi - lo) * i / 40.0, z=30.0 + oz) for i in range(40)]
    recs += [Receiver(x=10.0 * (nx // 2) + 13.0 * i + ox, z=(-7.0 if fs else 2.0) + oz) for i in range(-4, 5)]
    recs += [Receiver(x=10.0 * (nx // 2) + ox, z=10.0 * nz + hi - 20.0 + oz)]
    return recs


@pytest.mark.parametrize("pattern", ["x", "z", "both", "none"])
@pytest.mark.parametrize("nx,nz,pml,half,fs,nsrc", [(61, 47, 6, 4, True, 3), (64, 48, 10, 8, False, 1),
                                                    (77, 53, 11, 8, True, 2), (131, 203, 20, 4, False, 4)])
def test_traces_of_several_taps(nx, nz, pml, half, fs, nsrc, pattern):
    """Windows on one CTA's rows, across two, above the surface and on the sources' taps, against the step launches."""
    vp, rho = model(nz, nx)
    nt = 160
    s = SSGSolver(L.OWL_ACOUSTIC_ISO_2D, nx, nz, 10.0, 10.0, 1e-3, nt, pml=pml, fdhalf=half, free_surface=fs,
                  f0_max=12.0, max_shots=2)
    s.set_model(vp, rho)
    shots = [Shot(k + 1, [Source(x=10.0 * (nx // 2) + 7.3 * j, z=52.0 + 41.0 * j, f0=14.0 + j, t0=0.03 * j)
                          for j in range(nsrc)], spread(nx, nz, half, pml, fs, pattern)[k:]) for k in range(2)]
    ps = s.prepare(shots)
    a = s.forward(ps, RunOpts())
    assert s.last_info.gpu_launches < nt
    b = s.forward(ps, STEPWISE)
    assert s.last_info.gpu_launches > 2 * nt
    assert np.all(np.isfinite(b)) and np.abs(b).max() > 0
    np.testing.assert_array_equal(a, b)
    # the same with the traces recorded segment by segment, at the data sampling of a gradient's forward
    syn = np.zeros_like(b)
    s.gradient(ps, (0.5 * b).astype(np.float32), opts=RunOpts(checkpoint_interval=33), seis_out=syn)
    np.testing.assert_array_equal(syn, b)


@pytest.mark.parametrize("nx,nz,pml,half,nshots,forward,again", [
    (100, 80, 10, 4, 3, True, True),      # one wave
    (250, 150, 20, 4, 16, True, False),   # three waves: the storing segments are faster step by step
    (380, 180, 20, 8, 16, False, False),  # two passes a thread, three waves
])
def test_which_segments_run_resident(nx, nz, pml, half, nshots, forward, again):
    """Forward and recomputed segments are chosen apart; the run info tells which ran, and the results agree."""
    vp, rho = model(nz, nx)
    nt = 60
    s = SSGSolver(L.OWL_ACOUSTIC_ISO_2D, nx, nz, 10.0, 10.0, 1e-3, nt, pml=pml, fdhalf=half, f0_max=12.0,
                  max_shots=nshots)
    s.set_model(vp, rho)
    ps = s.prepare([Shot(k + 1, [Source(x=10.0 * nx * (k + 1) / (nshots + 1) + 3.3, z=61.7, f0=12.0)],
                         [Receiver(x=20.0 * i + 20.0, z=20.0) for i in range(20)]) for k in range(nshots)])
    b = s.forward(ps, STEPWISE)
    assert s.last_info.shots_per_cta_forward == 1 and s.last_info.tile_z_forward == 8
    a = s.forward(ps, RunOpts())
    info = s.last_info
    assert (info.shots_per_cta_forward < 0, info.gpu_launches < nt) == (forward, forward)
    if forward:
        np.testing.assert_array_equal(a, b)
        assert info.tile_z_forward == 0 and (info.tile_z, info.shots_per_cta) == (0, info.shots_per_cta_forward)
    else:
        close(a, b)
    obs = (0.5 * b).astype(np.float32)
    syn = np.zeros_like(b)
    _, g0 = s.gradient(ps, obs, opts=RunOpts(checkpoint_interval=20), seis_out=syn)
    assert (s.last_info.shots_per_cta_forward < 0) == forward
    assert (s.last_info.tile_z_forward == 0) == again
    np.testing.assert_array_equal(syn, a)  # the forward of a gradient runs as a forward alone
    _, g1 = s.gradient(ps, obs, opts=RunOpts(checkpoint_interval=20, use_graph=-1, tile_z=8, shots_per_cta=1))
    for p in range(2):
        close(np.split(g0, 2)[p], np.split(g1, 2)[p])
