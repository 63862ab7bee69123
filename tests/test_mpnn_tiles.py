"""The network's training pass on tiles of whole nodes (message sums in the edge
MLP's epilogue, edge adjoints summed in the backward tile) against the path
that stores both per edge (KFUN3D_MPNN_FUSED=0).

The forward sums are the same bit for bit, so the loss is; the adjoints are
added per node in another order in FP32 and then rounded to BF16 for the next
product, so the gradients may differ by a few BF16 units (2^-8) of their norm.
Sizes: one partial tile, several tiles, more tiles than CTAs.
"""
import numpy as np
import pytest

import kfun3d_b200 as kf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3, 9, 24])
def test_tiled_training_pass_matches_the_per_edge_one(box_mesh, monkeypatch, n):
    import torch
    from kfun3d_b200 import learned
    m = kf.Mesh(box_mesh(n, seed=51))
    N = m.nnodes
    rng = np.random.default_rng(n)
    x0 = torch.from_numpy(np.concatenate([rng.standard_normal((N, 4)), m.view.q.reshape(-1, 4)], axis=1))
    x0 = x0.to(device="cuda", dtype=torch.bfloat16)
    tgt = torch.from_numpy(rng.standard_normal((N, 4)).astype(np.float32)).cuda()
    res = []
    for fused in ("1", "0"):
        monkeypatch.setenv("KFUN3D_MPNN_FUSED", fused)
        net, graph = learned.Network(seed=4), learned.Graph(m)
        th = net.params()
        o, k, nr, off = learned.layer_shapes()[15]
        th[off:off + o * k] *= 10.0
        net.set_params(th)
        net.zero_grad()
        loss = net.accumulate(graph, x0, tgt, 1.0 / (4 * N))
        res.append((loss, net.grad().astype(np.float64)))
    (l0, g0), (l1, g1) = res
    assert l0 == l1 and np.all(np.isfinite(g0)) and np.linalg.norm(g0) > 0
    assert np.linalg.norm(g0 - g1) <= 4 * 2.0 ** -8 * np.linalg.norm(g1)
