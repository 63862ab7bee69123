"""A solve uses the factor of the precision that is set, whatever was factored or
solved in between: FP64 and FP32 factors of one mesh are both held, though the
sweeps' packed copy has room for one.

Both host and device entry points give, bit for bit, what they gave before a
whole solve in the other precision; the sizes are one that takes eight lanes a
row and one (from 150,000 rows) that takes four.  An FP64 solve after a fill
without a factorisation reads the matrix as it stands, as the level launches
(KFUN3D_SPTRSV=pdl4) do.
"""
import ctypes as C

import numpy as np
import pytest

import kfun3d_b200 as kf
from conftest import seeded_state
from kfun3d_b200.geometry import GEOMETRY
from oracle import port

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _settings(monkeypatch):
    kf.set_mode("fast")
    kf.set_aoa(3.06)
    monkeypatch.delenv("KFUN3D_SPTRSV", raising=False)
    yield
    kf.set_mode("exact")
    kf.set_precision(0)
    kf.set_ilu_order(0)
    kf.set_aoa(3.0)


def noalloc(m, b):
    import torch
    f = kf.lib().kfun3d_sptrsv_device_noalloc
    f.restype, f.argtypes = C.c_int, [C.POINTER(GEOMETRY), C.c_void_p, C.c_void_p]
    db = torch.from_numpy(b).to("cuda")
    dx = torch.full_like(db, float("nan"))
    rc = f(m.g, db.data_ptr(), dx.data_ptr())
    assert rc == 0, kf.last_error()
    return dx.cpu().numpy()


def mesh_state(box_mesh, n):
    m = kf.Mesh(box_mesh(n, seed=61))
    v = m.view
    q = seeded_state(v.q.copy(), 61)
    return m, q, port.timestep(m.g, v.nnodes, 40.0, q), np.random.default_rng(n).standard_normal(v.dofs)


@pytest.mark.parametrize("order", [0, 1])
@pytest.mark.parametrize("first", [0, 1])
@pytest.mark.parametrize("n", [9, 54])
def test_a_factor_outlives_work_in_the_other_precision(box_mesh, n, first, order):
    m, q, cdt, b = mesh_state(box_mesh, n)
    kf.set_ilu_order(order)
    kf.set_precision(first)
    m.fill(q, cdt)
    m.ilu()
    solves = [lambda: m.sptrsv(b)] + ([lambda: noalloc(m, b)] if order == 0 else [])
    for solve in solves:
        before = solve()
        kf.set_precision(1 - first)
        m.solve(ts_max=1)
        kf.set_precision(first)
        assert np.array_equal(solve(), before)
        # and the other precision's factor after this one's solves
        kf.set_precision(1 - first)
        other = m.sptrsv(b)
        kf.set_precision(first)
        assert np.array_equal(solve(), before)
        kf.set_precision(1 - first)
        assert np.array_equal(m.sptrsv(b), other)
        kf.set_precision(first)
        assert np.all(np.isfinite(before)) and np.linalg.norm(other - before) > 0
    m.close()


def test_fp64_solve_reads_the_matrix_as_it_stands(box_mesh, monkeypatch):
    res = []
    for sched in (None, "pdl4"):
        if sched:
            monkeypatch.setenv("KFUN3D_SPTRSV", sched)
        m, q, cdt, b = mesh_state(box_mesh, 9)
        m.fill(q, cdt)
        m.ilu()
        factor = m.sptrsv(b)
        m.fill(q, cdt)
        res.append(m.sptrsv(b))
        m.close()
        assert not np.array_equal(res[-1], factor)
    assert np.array_equal(res[0], res[1], equal_nan=True)
