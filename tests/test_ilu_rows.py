"""ILU(0) levels with a row's operands staged through shared memory (the
default) against the kernels that serve rows too long for that
(KFUN3D_ILU=pairs): the same factor bit for bit, in both precisions and both
elimination orders, on two factorisations in a row (the second starts from the
first's persistent L slots).

Sizes: fewer rows than a CTA takes, rows without lower blocks, rows whose
products fill one, two and three batches of 16.
"""
import numpy as np
import pytest

import kfun3d_b200 as kf
from conftest import seeded_state
from oracle import port

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["exact", "fast"])
@pytest.mark.parametrize("n", [3, 8, 21])
def test_staged_rows_equal_the_pair_kernels(box_mesh, monkeypatch, n, mode):
    kf.set_mode(mode)
    kf.set_aoa(3.06)
    path = box_mesh(n, seed=47)
    res = {}
    try:
        for kind in ("rows", "pairs"):
            if kind == "pairs":
                monkeypatch.setenv("KFUN3D_ILU", "pairs")
            m = kf.Mesh(path)
            v = m.view
            q = seeded_state(v.q.copy(), 47)
            cdt = port.timestep(m.g, v.nnodes, 40.0, q)
            b = np.random.default_rng(n).standard_normal(v.dofs)
            for order in (0, 1):
                kf.set_ilu_order(order)
                for prec in (0, 1):
                    kf.set_precision(prec)
                    for step in range(2):
                        m.fill(q + 0.01 * step, cdt)
                        m.ilu()
                        res[kind, order, prec, step] = m.sptrsv(b) if order else m.matrix()[2].copy()
                        assert kf.last_status() == 0, kf.last_error()
            kf.set_ilu_order(0)
            m.close()
    finally:
        kf.set_mode("exact")
        kf.set_precision(0)
        kf.set_ilu_order(0)
        kf.set_aoa(3.0)
    for key, x in res.items():
        if key[0] == "rows":
            assert np.all(np.isfinite(x)) and np.array_equal(x, res[("pairs",) + key[1:]]), key
