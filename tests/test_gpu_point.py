"""The point kernels at the trace and node counts where their CTAs per shot
change (1, a cluster of 2, 4 or 8, more with a launch per phase), sources'
and traces' taps overlapping: traces against the same receivers modelled in
groups of one CTA, to the bit; source-side adjoints of the separate point kernel
against the stencil kernels' own scatter, to the bit, and the FP64 oracle."""
import os

import numpy as np
import pytest

import oracle
from owl_b200 import _lib as L
from owl_b200.geometry import GridSpec, PreparedShots, Receiver, Shot, Source
from owl_b200.solver import RunOpts

from cases import desc, prepare, random_model, rel
from test_gpu_ac2d import make_solver
from test_gpu_ac3d import case3, solver3
from test_gpu_el2d import make
from test_oracle_el2d import DX, NX, NZ, el_desc, el_model

pytestmark = pytest.mark.gpu


def receivers(n, lo, hi, seed):
    """n of them between the nodes, the first ones around the sources"""
    rng = np.random.default_rng(seed)
    p = lo + (hi - lo) * rng.random((n, 3))
    return [Receiver(x=float(a), y=float(b), z=float(c), weight=float(w)) for (a, b, c), w in
            zip(p, rng.choice([1.0, 0.7], n))]


def forward(medium, recs):
    if medium == "ac3d":
        d, vp, rho, _ = case3(nt=40)
        s = solver3(d, vp, rho)
        src = [Source(x=123.3, y=101.7, z=91.2, f0=20.0), Source(x=127.0, y=99.0, z=95.5, f0=17.0, amp=0.6),
               Source(x=90.0, y=80.0, z=100.0, f0=18.0, mechanism="force", polar=35.0, azimuth=20.0)]
        grid = GridSpec(nx=d.nx, nz=d.nz, dx=d.dx, dz=d.dx, ny=d.ny, dy=d.dx)
        ps = PreparedShots([Shot(1, src, recs), Shot(2, src[:1], recs[: len(recs) // 2])], grid, d.dt)
        ncomp, opts = 1, RunOpts(tile_z=2)
    else:
        d = el_desc(0, L.OWL_ANISO_ISO)
        s = make(d, el_model(L.OWL_ANISO_ISO))
        src = [Source(x=0.5 * NX * DX + 3.0, z=0.5 * NZ * DX, f0=20.0),
               Source(x=0.5 * NX * DX - 8.0, z=0.5 * NZ * DX + 5.0, f0=18.0, mechanism="force", polar=30.0)]
        ps = s.prepare([Shot(1, src, recs), Shot(2, src[:1], recs[: len(recs) // 2])])
        ncomp, opts = 2, RunOpts(tile_z=8, shots_per_cta=1)
    out = s.forward(ps, opts)
    n0 = ncomp * len(recs) * d.nt
    return out[:n0].reshape(ncomp, len(recs), -1), out[n0:].reshape(ncomp, len(recs) // 2, -1)


@pytest.mark.parametrize("medium,n", [("ac3d", 300), ("ac3d", 700), ("ac3d", 1500), ("ac3d", 2500),
                                      ("el2d", 140), ("el2d", 400), ("el2d", 900), ("el2d", 1300)])
def test_traces_of_many_ctas_equal_those_of_one(medium, n):
    recs = receivers(n, 60.0, 150.0, n) if medium == "ac3d" else receivers(n, 0.3 * NX * DX, 0.7 * NX * DX, n)
    a, b = forward(medium, recs)
    assert np.all(np.isfinite(a)) and np.abs(a).max() > 0
    per = 128 if medium == "ac3d" else 64
    for i in range(0, n, 2 * per):
        # (the second shot's half of each group of 2 per receivers is its first per ones)
        ga, gb = forward(medium, recs[i:i + 2 * per])
        np.testing.assert_array_equal(a[:, i:i + 2 * per], ga)
        m = min(gb.shape[1], max(0, b.shape[1] - i))
        np.testing.assert_array_equal(b[:, i:i + m], gb[:, :m])


@pytest.mark.parametrize("n", [2, 5, 11, 24, 150])
def test_source_adjoint_after_a_scatter_of_many_ctas(n):
    nx, nz, dx, dt, nt = 120, 100, 10.0, 1e-3, 80
    d = desc(nx, nz, dx, dt, nt)
    vp, rho = random_model(nx, nz)
    rng = np.random.default_rng(n)
    # the first receiver's window meets both sources' taps; the others apart from each other while they fit
    recs = [Receiver(x=612.3, z=498.7)] + [Receiver(x=110.0 + 97.0 * (i % 11) + 5.0 * rng.random() + 2.0,
                                                    z=105.0 + 93.0 * (i // 11 % 9) + 5.0 * rng.random() + 2.0) for i in range(n - 1)]
    src = [Source(x=603.3, z=501.7, f0=15.0), Source(x=620.0, z=480.4, f0=12.0, amp=0.5)]
    ps = prepare([Shot(1, src, recs), Shot(2, src[1:], recs[:1])], nx, nz, dx, dt)
    s = make_solver(d, vp, rho)
    adj = rng.standard_normal(s.seis_size(ps)).astype(np.float32)
    opts = RunOpts(checkpoint_interval=20, tile_z=8, shots_per_cta=1)
    fused = s.source_gradient(ps, adj, opts)
    os.environ["OWL_FUSE"] = "0"
    try:
        got = s.source_gradient(ps, adj, opts)
        _, g = s.gradient(ps, adj, L.OWL_ADJ_GIVEN, opts)
    finally:
        os.environ.pop("OWL_FUSE", None)
    np.testing.assert_array_equal(got, fused)
    _, gref, sref = oracle.ac2d_gradient(d, vp, rho, ps, adj, adj_kind=L.OWL_ADJ_GIVEN, k=20, stf_grad=True)
    assert rel(g, gref) < 1e-4
    mask, off = np.zeros(sref.shape, dtype=bool), 0
    for sh in range(ps.nshots):
        for k in range(ps.arr[sh].nsrc):
            q = ps.arr[sh].src[k]
            mask[off + max(1, q.nbeg) - 1:off + min(nt, q.nbeg + q.nt_stf - 1)] = True
            off += nt
    assert mask.any() and rel(got[mask], sref[mask]) < 1e-4
