"""Fast mode's Gram-Schmidt (all projections from one pass over the basis)
against exact mode's sequential one: the same GMRES iterations, and per-step
residual norms that differ by no more than the two modes' rounding.  There the
basis is orthonormal to rounding; one column against a basis that is not, whose
Gram matrix the fast form has to take into account, is compared with the
sequential sweep in 80-bit arithmetic.

Sizes of the solves: fewer elements than a CTA has threads, a few CTAs, restart
cycles (more than 30 iterations a step).  Of the columns: also grids past the
296 CTAs of the products and the update (from 37,888 nodes) and past the 1,184
of the scaling (from 151,552), and more basis vectors than a pass takes at once
(8).
The bound on the norms, 1e-3, is what two builds of the reference that differ
in contraction only show (up to 9.4e-4 per step on its own small mesh: the norm
after an inexact step amplifies rounding); a projection left out or applied
twice changes the iteration counts and the norms by far more.
"""
import numpy as np
import pytest

import kfun3d_b200 as kf
from kfun3d_b200 import api

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


def skewed_basis(dofs, count):
    """Unit vectors with a common part (every product of two about 0.2)."""
    rng = np.random.default_rng(dofs)
    V = rng.standard_normal((count, dofs))
    V /= np.linalg.norm(V, axis=1)[:, None]
    V[1:] += 0.5 * V[0]
    return V / np.linalg.norm(V, axis=1)[:, None]


@pytest.mark.parametrize("mode", ["exact", "fast"])
@pytest.mark.parametrize("n,last", [(3, 16), (12, 16), (35, 9), (54, 9)])
def test_column_against_a_basis_that_is_not_orthonormal(box_mesh, n, last, mode):
    kf.set_mode(mode)
    try:
        m = kf.Mesh(box_mesh(n, seed=43))
        V = skewed_basis(m.view.dofs, last + 2)
        for k in range(last + 1):
            buf, h = V[:k + 2].copy(), np.zeros(k + 2)
            assert kf.lib().kfun3d_gram_schmidt(m.g, k, api._d(buf), api._d(h)) == 0, kf.last_error()
            if k not in (0, 1, 7, 8, last):
                continue
            B = V[:k + 1].astype(np.longdouble)
            w = V[k + 1].astype(np.longdouble)
            ref = np.zeros(k + 2, dtype=np.longdouble)
            for v in range(k + 1):
                ref[v] = B[v] @ w
                w = w - ref[v] * B[v]
            ref[k + 1] = np.sqrt(w @ w)
            # a product of two unit vectors is off by at most `depth` roundings
            # (the longest chain of additions: in index order, or a thread's
            # share and the trees above it); (I + L) h = V^T w passes the
            # errors of L and V^T w on to h by its inverse's magnitudes
            eps, depth = 2.0 ** -53, m.view.dofs if mode == "exact" else 64
            L = np.tril(np.abs((B @ B.T).astype(np.float64)), -1)
            inv = np.linalg.inv(np.eye(k + 1) - L)
            err = inv.sum(1) * (k + 2) * depth * eps * (1.0 + np.abs(ref[:-1]).sum())
            assert np.all(np.abs(h[:-1] - ref[:-1]) <= err), (k, h[:-1] - ref[:-1], err)
            moved = err.sum() + (k + 2) * eps * (1.0 + np.abs(ref).sum())   # of w, in norm
            assert abs(h[-1] - ref[-1]) <= moved + depth * eps
            assert np.linalg.norm((buf[k + 1] - w / ref[-1]).astype(np.float64)) <= 4 * (moved + depth * eps) / ref[-1]
            assert np.max(err) < 1e-3 * np.max(np.abs(ref[:-1]))   # far below what the basis' products contribute
        m.close()
    finally:
        kf.set_mode("exact")
