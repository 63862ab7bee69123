"""The gradient with its incidence staged in shared memory (the default) against
the one that reads it from global memory (KFUN3D_GRADIENT=plain), which serves
meshes whose widest range of 64 nodes does not fit: the same gradients and the
same residual bit for bit, in both node orders; in exact mode they do not
depend on the node order, and the residual equals the oracle's.

Sizes: fewer nodes than a CTA takes (27), just under and over a multiple of 64
(125 and 729), a multiple (512).
"""
import numpy as np
import pytest

import kfun3d_b200 as kf
from conftest import seeded_state
from oracle import port

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["exact", "fast"])
@pytest.mark.parametrize("n", [3, 5, 8, 9])
def test_staged_gradient_equals_the_plain_one(box_mesh, monkeypatch, n, mode):
    kf.set_mode(mode)
    kf.set_aoa(3.06)
    path = box_mesh(n, seed=53)
    res = {}
    try:
        for order in ("natural", "morton"):
            monkeypatch.setenv("KFUN3D_NODE_ORDER", order)
            for kind in ("tma", "plain"):
                monkeypatch.setenv("KFUN3D_GRADIENT", kind)
                m = kf.Mesh(path)
                q = seeded_state(m.view.q.copy(), 53)
                for fo in (0, 1):
                    kf.set_first_order(fo)
                    grads, r = m.flux(q)
                    assert kf.last_status() == 0, kf.last_error()
                    res[order, kind, fo] = [*grads, r]
                    if mode == "exact":
                        assert np.array_equal(r, port.flux(m.g, 3.06, q, first_order=bool(fo))[1])
                m.close()
    finally:
        kf.set_mode("exact")
        kf.set_first_order(0)
        kf.set_aoa(3.0)
    for (order, kind, fo), got in res.items():
        for a, b in zip(got, res["natural" if mode == "exact" else order, "plain", fo]):
            assert np.all(np.isfinite(a)) and np.array_equal(a, b), (order, kind, fo)
