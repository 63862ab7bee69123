"""Large host arrays go to and from the device through pinned buffers filled by
several threads; arrays that are pinned already are copied directly.  The same
residual and gradients bit for bit either way, on calls in a row (the buffers
are used again), with last chunks that are not full.

Sizes: 34 (1 MB in and 5 MB out, both copied directly), 66 (9 MB in directly,
37 MB out staged), 102 (34 MB in, 136 MB out, both staged: each call's copies
out take the buffers that its copies in may still be leaving).
"""
import ctypes as C

import numpy as np
import pytest
import torch

import kfun3d_b200 as kf
from conftest import seeded_state
from kfun3d_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [34, 66, 102])
def test_pageable_arrays_equal_pinned_ones(box_mesh, n):
    kf.set_mode("fast")
    try:
        m = kf.Mesh(box_mesh(n, seed=59))
        for seed in (1, 2, 3):
            q = seeded_state(m.view.q.copy(), seed)
            grads, r = m.flux(q)
            pin = [torch.zeros(q.size, dtype=torch.float64).pin_memory().numpy() for _ in range(5)]
            pin[0][:] = q
            grad = api.GRADIENT(*(api._d(x) for x in pin[1:4]))
            kf.lib().ComputeFlux(m.g, api._d(pin[0]), C.byref(grad), api._d(pin[4]))
            assert kf.last_status() == 0, kf.last_error()
            for a, b in zip((*grads, r), pin[1:]):
                assert np.any(a != 0.0) and np.array_equal(a, b)
        m.close()
    finally:
        kf.set_mode("exact")
