"""Fast mode's Gram-Schmidt (all projections from one pass over the basis)
against exact mode's sequential one: the same GMRES iterations, and per-step
residual norms that differ by no more than the two modes' rounding.

Sizes: fewer elements than a CTA has threads, grids short of the full 296
blocks and past it, restart cycles (more than 30 iterations a step).
The bound on the norms, 1e-3, is what two builds of the reference that differ
in contraction only show (up to 9.4e-4 per step on its own small mesh: the norm
after an inexact step amplifies rounding); a projection left out or applied
twice changes the iteration counts and the norms by far more.
"""
import numpy as np
import pytest

import kfun3d_b200 as kf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,restart", [(3, 30), (7, 30), (12, 30), (12, 7), (16, 1)])
def test_fast_gram_schmidt_follows_the_sequential_sweep(box_mesh, n, restart):
    path = box_mesh(n, seed=43)
    hist = {}
    kf.set_aoa(3.06)
    try:
        for mode in ("exact", "fast"):
            kf.set_mode(mode)
            m = kf.Mesh(path)
            m.reset_state()
            hist[mode] = m.solve(ts_max=4, gmres_restart=restart, gmres_rtol=1e-3, gmres_max_it=400)
            m.close()
    finally:
        kf.set_mode("exact")
        kf.set_aoa(3.0)
    assert kf.last_status() == 0
    assert [s["gmres_its"] for s in hist["fast"]] == [s["gmres_its"] for s in hist["exact"]]
    a = np.array([s["fnorm"] for s in hist["fast"]])
    b = np.array([s["fnorm"] for s in hist["exact"]])
    assert np.all(np.abs(a - b) <= 1e-3 * b), (a, b)
