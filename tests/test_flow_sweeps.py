"""The data-flow triangular sweeps (the default schedule): both sweeps in one
launch, every row waiting for the values it reads.

Bit for bit the level launches' results (KFUN3D_SPTRSV=pdl4, the reference's
arithmetic per row, in both elimination orders) at the sizes where the chunking can go wrong: fewer rows
than a warp takes, chunks that end inside a level, eight lanes a row and (from
150,000 rows) four; several solves in a row, which alternate between the two
solution buffers; right-hand sides with NaN and infinities, whose bits are also
the sweeps' "not written" mark.
"""
import numpy as np
import pytest

import kfun3d_b200 as kf
from conftest import seeded_state
from oracle import port

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _settings(monkeypatch):
    kf.set_mode("fast")
    kf.set_aoa(3.06)
    monkeypatch.delenv("KFUN3D_SPTRSV", raising=False)
    monkeypatch.delenv("KFUN3D_ILU_PERM", raising=False)
    yield
    kf.set_mode("exact")
    kf.set_precision(0)
    kf.set_ilu_order(0)
    kf.set_aoa(3.0)


def right_hand_sides(dofs):
    rng = np.random.default_rng(dofs)
    out = [rng.standard_normal(dofs) for _ in range(3)]
    bad = rng.standard_normal(dofs)
    bad[dofs // 3] = np.array([-1], dtype=np.int64).view(np.float64)[0]   # the all-ones NaN
    bad[dofs // 2] = np.inf
    return out + [bad, out[0]]


@pytest.mark.parametrize("n", [3, 4, 9, 14, 31, 54])
def test_flow_sweeps_equal_level_launches(box_mesh, monkeypatch, n):
    path = box_mesh(n, seed=41)
    res = {}
    for sched in ("flow", "levels"):
        if sched == "levels":
            monkeypatch.setenv("KFUN3D_SPTRSV", "pdl4")
        m = kf.Mesh(path)
        v = m.view
        q = seeded_state(v.q.copy(), 41)
        cdt = port.timestep(m.g, v.nnodes, 40.0, q)
        for order in (0, 1):
            kf.set_ilu_order(order)
            for prec in (0, 1):
                kf.set_precision(prec)
                m.fill(q, cdt)
                m.ilu()
                assert m.query("sptrsv_flow") == (sched == "flow"), (sched, order)
                res[sched, order, prec] = [m.sptrsv(b) for b in right_hand_sides(v.dofs)]
                assert kf.last_status() == 0, (sched, order, prec, kf.last_error())
        m.close()
    for order in (0, 1):
        for prec in (0, 1):
            for k, (a, b) in enumerate(zip(res["flow", order, prec], res["levels", order, prec])):
                assert np.array_equal(a, b, equal_nan=True), (order, prec, k)
