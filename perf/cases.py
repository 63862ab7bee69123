"""Performance cases: the calls a user of kfun3d_b200 makes, over their real range of sizes and options.

A case is a seeded Kuhn-box mesh of n^3 nodes and one call, or one short
sequence of calls, through the package's public entry points:

  residual   Mesh.flux on host arrays (gradients and residual), as a host
             solver that keeps its own Newton loop calls it
  precond    Mesh.timestep, fill, ilu and sptrsv in sequence: one refresh of
             the preconditioner and one application of it
  trisolve   kfun3d_sptrsv_device_noalloc on device arrays, with a factor kept
             from earlier calls: a host framework's own Krylov iteration
  solve      Mesh.solve: the pseudo-transient Newton-GMRES solve
  flexible   Mesh.solve_flexible, without or with the shipped network
  network    Network.apply on device vectors: one learned correction
  train      one batch of the network's training: forward and backward of two
             pairs, the summed gradient and the loss returned

The mesh and its device mirror, the factor (trisolve) and the network are what
a program keeps between calls; the state, the right-hand sides and the angle
of attack come from the seed.
"""
import ctypes
import math
import os
import tempfile

import numpy as np
import torch

import kfun3d_b200 as kf
from kfun3d_b200 import learned

BETA = 15.0
CFL = 200.0


def _case(name, kind, n, mode="fast", precision="fp64", order="mesh", numbering=1, bump=0.1, aoa=3.06,
          first_order=False, network=False, mesh_seed=3):
    c = dict(kind=kind, n=n, mode=mode, precision=precision, order=order, numbering=numbering, bump=bump, aoa=aoa,
             first_order=first_order, network=network, mesh_seed=mesh_seed)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: one residual of a 1,000-node mesh in the library's
        # default arithmetic (the reference's own); latency and launches
        _case("residual_box10_exact", "residual", 10, mode="exact"),
        # one residual of the 343,000-node workload on host arrays
        _case("residual_box70", "residual", 70),
        # a preconditioner refresh on the 15,625-node CPU-runnable workload,
        # numbered along a space-filling curve as mesh generators write them
        _case("precond_box25_fp64", "precond", 25, numbering=2),
        # the same in mixed precision and the spatial elimination order on an
        # odd size between the workloads
        _case("precond_box63_mixed", "precond", 63, precision="fp32", order="spatial"),
        # a host framework applying the FP64 factor of the 343,000-node mesh to
        # its own device vectors, once per Krylov iteration
        _case("trisolve_box70_fp64", "trisolve", 70),
        # whole solves with the reference's parameters: a small mesh in the
        # default arithmetic, as parity runs use it
        _case("solve_box10_exact", "solve", 10, mode="exact"),
        # the CPU-runnable workload's mesh, FP64: launch-bound iterations
        _case("solve_box25_fp64", "solve", 25),
        # the plain FP64 workload
        _case("solve_box70_fp64", "solve", 70),
        # a mesh of the training workload solved with the shipped network
        _case("flexible_box40_network", "flexible", 40, precision="fp32", order="spatial", network=True),
        # the largest workload: 1.73 million nodes, mixed precision and the
        # spatial order (bump and angle of attack held out of training)
        _case("flexible_box120_mixed", "flexible", 120, precision="fp32", order="spatial", bump=0.12, aoa=4.5),
        # one learned correction of a Krylov vector
        _case("network_box70", "network", 70, network=True),
        # the training workload: a batch of two pairs on a 64,000-node mesh
        _case("train_box40", "train", 40, network=True),
    ]


# range of n for drawn cases; each costs less than the largest listed case
RANGE = {"residual": (8, 90), "precond": (8, 80), "trisolve": (8, 90), "solve": (8, 66), "flexible": (8, 66),
         "network": (8, 80), "train": (8, 44)}


def draw(rng):
    kind = rng.choice(["residual", "precond", "trisolve", "solve", "solve", "flexible", "flexible", "network", "train"])
    lo, hi = RANGE[kind]
    mode = "exact" if kind in ("residual", "precond", "solve") and rng.random() < 0.25 else "fast"
    if kind == "solve" and mode == "exact":
        hi = 13   # the default arithmetic sums in index order: small meshes in practice
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    learned_kind = kind in ("network", "train")
    order = rng.choice(["mesh", "spatial"]) if kind in ("precond", "solve", "flexible") and mode == "fast" else "mesh"
    precision = rng.choice(["fp64", "fp32"]) if kind in ("precond", "trisolve", "solve", "flexible") and mode == "fast" else "fp64"
    return _case(None, kind, n, mode=mode, precision=precision, order=order, numbering=rng.choice([1, 1, 2]),
                 bump=round(rng.uniform(0.05, 0.15), 4), aoa=round(rng.uniform(0.5, 6.0), 3),
                 first_order=kind == "residual" and rng.random() < 0.25,
                 network=learned_kind or (kind == "flexible" and rng.random() < 0.5),
                 mesh_seed=rng.randrange(1, 1 << 20))


# ---------------------------------------------------------------- state

_kept = {}   # the mesh of the last case, with what a program keeps beside it


def _mesh(case):
    key = tuple(case[k] for k in ("n", "numbering", "bump", "mesh_seed"))
    if _kept.get("key") != key:
        _kept.clear()
        with tempfile.TemporaryDirectory() as d:
            path = os.path.join(d, "box.msh")
            # numbering: 1 seeded random, 2 Morton order of the lattice
            kf.generate_mesh(path, case["n"], bump_height=case["bump"], seed=case["mesh_seed"], permute=case["numbering"])
            _kept.update(key=key, mesh=kf.Mesh(path))
    return _kept["mesh"]


def _settings(case, aoa):
    kf.set_mode(case["mode"])
    kf.set_precision(case["precision"])
    kf.set_ilu_order(case["order"])
    kf.set_first_order(case["first_order"])
    kf.set_aoa(aoa)


def _state(case, seed):
    """Angle of attack near the case's, and a flow state near its free stream."""
    rng = np.random.default_rng([seed, case["n"]])
    aoa = case["aoa"] + rng.uniform(-0.4, 0.4)
    a = aoa * math.pi / 180.0
    free = np.array([1.0, math.cos(a), math.sin(a), 0.0])
    q = np.tile(free, case["n"] ** 3)
    if case["kind"] not in ("solve", "flexible"):   # solves start from the free stream itself
        q += rng.uniform(-0.05, 0.05, q.size)
    return aoa, q, rng


def _weights():
    return np.load(os.path.join(os.path.dirname(kf.__file__), "weights", "mpnn_box40.npy"))


def _device_solve():
    """kfun3d_sptrsv_device_noalloc(GEOMETRY *, const double *d_b, double *d_x), declared as in the C header."""
    proto = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p)
    return proto(("kfun3d_sptrsv_device_noalloc", kf.lib()))


def _network():
    if "net" not in _kept:
        _kept["net"] = learned.Network(params=_weights())
    return _kept["net"]


def prepare(case, seed):
    m = _mesh(case)
    aoa, q, rng = _state(case, seed)
    s = dict(case=case, mesh=m, aoa=aoa, q=q)
    _settings(case, aoa)
    kind = case["kind"]
    if kind in ("network", "train"):
        if "graph" not in _kept:
            _kept["graph"] = learned.Graph(m)
        s["graph"], s["net"] = _kept["graph"], _network()
        if kind == "network":
            s["y"] = torch.from_numpy(0.01 * rng.standard_normal(q.size)).cuda()
            s["q_dev"] = torch.from_numpy(q).cuda()
        else:
            s["pairs"] = _pairs(case, q, rng, "cuda")
        return s
    plan = (kind, case["precision"], case["order"], case["aoa"])
    if _kept.get("plan") != plan:
        m.flux(q)   # the device mirror and the elimination order are built
        if kind == "trisolve":
            aoa_f, q_f, _ = _state(case, 0)   # the factor a framework keeps: that of a state of its own
            kf.set_aoa(aoa_f)
            m.timestep(CFL, q_f)
            m.fill()
            m.ilu()
        _kept["plan"] = plan
    if kind in ("precond", "trisolve"):
        s["b"] = rng.standard_normal(q.size)
    if kind == "trisolve":
        s["b_dev"] = torch.from_numpy(s["b"]).cuda()
        s["x_dev"] = torch.empty_like(s["b_dev"])
        s["solve"] = _device_solve()
    if kind == "flexible" and case["network"]:
        s["net"] = _network()
    return s


def _pairs(case, q, rng, device):
    """Two training pairs: features [y/s, q] in BF16 and FP32 targets."""
    pairs = []
    for _ in range(2):
        y = rng.standard_normal((q.size // 4, 4))
        x0 = torch.from_numpy(np.concatenate([y, q.reshape(-1, 4)], axis=1)).to(device=device, dtype=torch.bfloat16)
        t = torch.from_numpy(0.5 * rng.standard_normal((q.size // 4, 4))).to(device=device, dtype=torch.float32)
        pairs.append((x0, t))
    return pairs


def run(s):
    case, m, kind = s["case"], s["mesh"], s["case"]["kind"]
    _settings(case, s["aoa"])
    if kind == "residual":
        (gx, gy, gz), r = m.flux(s["q"])
        return {"gx": gx, "gy": gy, "gz": gz, "r": r}
    if kind == "precond":
        cdt = m.timestep(CFL, s["q"])
        m.fill()
        m.ilu()
        return {"cdt": cdt, "x": m.sptrsv(s["b"])}
    if kind == "trisolve":
        if s["solve"](ctypes.cast(m.g, ctypes.c_void_p), s["b_dev"].data_ptr(), s["x_dev"].data_ptr()) != 0:
            raise RuntimeError(kf.last_error())
        return {"x": s["x_dev"]}
    if kind in ("solve", "flexible"):
        m.view.q[:] = s["q"]
        if kind == "solve":
            h = m.solve()
        else:
            h, _ = m.solve_flexible(s.get("net"))
        return {"q": m.view.q, "forces": [h[-1]["lift"], h[-1]["drag"], h[-1]["momn"]]}
    if kind == "network":
        return {"z": s["net"].apply(s["graph"], s["y"], s["q_dev"])}
    net = s["net"]
    net.zero_grad()
    w = 1.0 / (len(s["pairs"]) * 4 * m.nnodes)
    loss = sum(net.accumulate(s["graph"], x0, t, w) for x0, t in s["pairs"])
    return {"loss": loss, "grad": net.grad()}


# ---------------------------------------------------------------- work and tolerance

def work(case):
    n = case["n"]
    N = n ** 3
    E = 3 * n * n * (n - 1) + 3 * n * (n - 1) ** 2 + (n - 1) ** 3
    nnz = N + 2 * E
    w = 4 if case["precision"] == "fp32" else 8
    kind = case["kind"]
    edges = 40 * E + 24 * N                    # end points, normals and areas; coordinates
    flux = edges + 48 * E + 64 * N             # with the least-squares terms, the state and the residual
    flux_flops = 330 * E
    trsv = nnz * (16 * w + 4) + 64 * N
    setup = (40 * E + 40 * N) + (40 * E + 40 * N + nnz * (16 * w + 4)) + 2 * nnz * 16 * w   # time step, fill, ILU(0)
    setup_flops = 450 * E + 128 * 14 * nnz
    if kind == "residual":
        if case["first_order"]:
            return {"bytes": edges + 64 * N, "flops": 260 * E}
        return {"bytes": flux + 96 * N, "flops": flux_flops}
    if kind == "precond":
        return {"bytes": setup + trsv, "flops": setup_flops + 32 * nnz}
    if kind == "trisolve":
        return {"bytes": trsv, "flops": 32 * nnz}
    if kind in ("solve", "flexible"):
        # GMRES iterations of a solve to the default 1e-7 drop, about, and the
        # basis vectors an iteration reads on average
        its = (6 if case["order"] == "spatial" else 9) * n
        per = flux + trsv + 32 * N * 15
        return {"bytes": its * per + 7 * setup, "flops": its * (flux_flops + 32 * nnz + 240 * N) + 7 * setup_flops}
    R = 2 * E
    flops = 2 * (R * 3 * (68 * 32 + 32 * 32) + N * (8 * 32 + 32 * 32 + 3 * (64 * 32 + 32 * 32) + 32 * 32 + 32 * 4))
    layer = R * 16 + N * 64 * 4                # an edge's indices and features; the node states and sums
    if kind == "network":
        return {"bytes": 3 * layer + 96 * N, "flops": flops}
    return {"bytes": 2 * (3 * 3 * layer + 96 * N), "flops": 2 * 3 * flops}


def tolerance(case):
    kind = case["kind"]
    if case["mode"] == "exact" and kind != "precond":
        return "exact"   # the reference's operation order: bit-identical by contract
    if kind == "residual":
        return {"rel": 5e-14, "max": 1e-11}   # 4e-15 from 64-bit sums in another order
    if kind in ("precond", "trisolve"):
        if case["precision"] == "fp32":
            return {"rel": 1e-6, "max": 1e-4}   # FP32 factors: 1.3e-7 from the FP64 factor's solve
        return {"rel": 1e-13, "max": 1e-11}
    if kind in ("solve", "flexible"):
        # stopped at a 1e-7 drop: another preconditioner moves the state by up
        # to 4e-10 and the forces (the lift is small) by up to 1.6e-8
        return {"rel": 6e-8, "max": 1e-7}
    # BF16 features and activations: 1.5e-2 from 64 bits, the gradient of
    # random targets (sums that cancel) up to 7e-2
    return {"rel": 1e-2, "max": 0.2} if kind == "network" else {"rel": 5e-2, "max": 0.5}


# ---------------------------------------------------------------- the same in 64 bits, plain torch

def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


class _Geo:
    """The mesh arrays as float64 / int64 tensors."""

    def __init__(self, v):
        d = _dev()
        f = lambda a: torch.from_numpy(np.array(a, dtype=np.float64)).to(d)              # noqa: E731
        i = lambda a: torch.from_numpy(np.array(a).astype(np.int64)).to(d)               # noqa: E731
        self.N, self.d = v.nnodes, d
        self.n0, self.n1 = i(v.n0), i(v.n1)
        self.nrm, self.area = torch.stack([f(v.xn), f(v.yn), f(v.zn)], 1), f(v.area)
        self.xyz = torch.stack([f(a) for a in v.xyz], 1)
        self.w0, self.w1 = torch.stack([f(a) for a in v.w0], 1), torch.stack([f(a) for a in v.w1], 1)
        self.s, self.sn = i(v.s_nodes), torch.stack([f(a) for a in v.s_xyz], 1)
        self.f, self.fn = i(v.f_nodes), torch.stack([f(a) for a in v.f_xyz], 1)
        self.face = torch.stack([i(a) for a in v.faces], 1)


def _flux_jacobian(q, n):
    """dF/dq of the artificial-compressibility flux through the unit normal n."""
    u, ub = q[:, 1:], (q[:, 1:] * n).sum(1)
    A = torch.zeros(len(q), 4, 4, dtype=torch.float64, device=q.device)
    A[:, 0, 1:] = BETA * n
    A[:, 1:, 0] = n
    A[:, 1:, 1:] = u[:, :, None] * n[:, None, :] + ub[:, None, None] * torch.eye(3, dtype=torch.float64, device=q.device)
    return A


def _projectors(q, n):
    """Spectral projectors of _flux_jacobian for ubar, ubar + c and ubar - c, and those eigenvalues."""
    A, ub = _flux_jacobian(q, n), (q[:, 1:] * n).sum(1)
    c = torch.sqrt(ub * ub + BETA)
    lam = [ub, ub + c, ub - c]
    eye = torch.eye(4, dtype=torch.float64, device=q.device)
    S = [A - l[:, None, None] * eye for l in lam]
    P = []
    for i in range(3):
        j, k = [t for t in range(3) if t != i]
        P.append(S[j] @ S[k] / ((lam[i] - lam[j]) * (lam[i] - lam[k]))[:, None, None])
    return P, lam


def _abs_jacobian(q, n):
    P, lam = _projectors(q, n)
    return sum(p * l.abs()[:, None, None] for p, l in zip(P, lam))


def _flux(q, n):
    ub = (q[:, 1:] * n).sum(1, keepdim=True)
    return torch.cat([BETA * ub, q[:, 1:] * ub + n * q[:, :1]], 1)


def _free(aoa, d):
    a = aoa * math.pi / 180.0
    return torch.tensor([[1.0, math.cos(a), math.sin(a), 0.0]], dtype=torch.float64, device=d)


def _farfield(G, q, aoa):
    """Far-field state, unit normal, area and d(state)/dq at the far-field nodes."""
    area = G.fn.norm(dim=1)
    n, qi = G.fn / area[:, None], q[G.f]
    free = _free(aoa, q.device).expand(len(qi), 4)
    P, _ = _projectors(free, n)
    out = ((qi[:, 1:] * n).sum(1) > 0)[:, None, None].double()
    dq = P[0] * out + P[1]
    qb = (dq @ qi[:, :, None] + (P[0] * (1 - out) + P[2]) @ free[:, :, None])[:, :, 0]
    return qb, n, area, dq


def _exact_residual(G, q, aoa, first_order):
    grad = torch.zeros(G.N, 3, 4, dtype=torch.float64, device=q.device)
    if not first_order:
        dq = (q[G.n1] - q[G.n0])[:, None, :]
        grad.index_add_(0, G.n0, G.w0[:, :, None] * dq)
        grad.index_add_(0, G.n1, G.w1[:, :, None] * -dq)
    xm = 0.5 * (G.xyz[G.n0] + G.xyz[G.n1])
    L, R = (q[k] + ((xm - G.xyz[k])[:, :, None] * grad[k]).sum(1) for k in (G.n0, G.n1))
    f = 0.5 * (_flux(L, G.nrm) + _flux(R, G.nrm) - (_abs_jacobian(0.5 * (L + R), G.nrm) @ (R - L)[:, :, None])[:, :, 0])
    f = f * G.area[:, None]
    r = torch.zeros_like(q)
    r.index_add_(0, G.n0, f)
    r.index_add_(0, G.n1, -f)
    x = [G.xyz[G.face[:, k]] for k in range(3)]
    wall = -torch.linalg.cross(x[1] - x[0], x[2] - x[0]) / 6.0
    p = [q[G.face[:, k], 0] for k in range(3)]
    for k in range(3):
        pk = 0.75 * p[k] + 0.125 * (p[(k + 1) % 3] + p[(k + 2) % 3])
        r.index_add_(0, G.face[:, k], torch.cat([torch.zeros_like(pk)[:, None], wall * pk[:, None]], 1))
    qb, n, area, _ = _farfield(G, q, aoa)
    r.index_add_(0, G.f, _flux(qb, n) * area[:, None])
    return grad, r


def _exact_timestep(G, q):
    acc = torch.zeros(G.N, dtype=torch.float64, device=q.device)

    def add(node, u, n, area):
        ub = (u * n).sum(1)
        term = (ub.abs() + torch.sqrt(ub * ub + BETA)) * area
        for k in node:
            acc.index_add_(0, k, term)
    add((G.n0, G.n1), 0.5 * (q[G.n0, 1:] + q[G.n1, 1:]), G.nrm, G.area)
    for node, nv in ((G.s, G.sn), (G.f, G.fn)):
        ln = nv.norm(dim=1)
        add((node,), q[node, 1:], nv / ln[:, None], ln)
    return acc / CFL


def _exact_factor_solve(G, q, aoa, cdt, rank, b):
    """(LU)^-1 b for the block ILU(0) factor of the first-order Jacobian in the elimination order `rank`."""
    d, N = q.device, G.N
    qa, qb = q[G.n0], q[G.n1]
    ab = _abs_jacobian(0.5 * (qa + qb), G.nrm)
    h = (0.5 * G.area)[:, None, None]
    v0, v1 = h * (_flux_jacobian(qa, G.nrm) + ab), h * (_flux_jacobian(qb, G.nrm) - ab)
    D = cdt[:, None, None] * torch.eye(4, dtype=torch.float64, device=d)
    D.index_add_(0, G.n0, v0)
    D.index_add_(0, G.n1, -v1)
    D[:, 1:, 0].index_add_(0, G.s, G.sn)
    far, n, area, dq = _farfield(G, q, aoa)
    D.index_add_(0, G.f, area[:, None, None] * (_flux_jacobian(far, n) @ dq))
    rank = rank.to(d)
    r0, r1, ids = rank[G.n0], rank[G.n1], rank
    key = torch.cat([ids * N + ids, r0 * N + r1, r1 * N + r0])
    key, perm = key.sort()
    A = torch.cat([D, v1, -v0])[perm]
    row, col = key // N, key % N
    ia = torch.searchsorted(row, torch.arange(N + 1, device=d))
    diag = torch.searchsorted(key, torch.arange(N, device=d) * (N + 1))

    def levels(mask):
        lev, r, c = torch.zeros(N, dtype=torch.int64, device=d), row[mask], col[mask]
        while True:
            new = torch.zeros_like(lev).scatter_reduce_(0, r, lev[c] + 1, "amax")
            if torch.equal(new, lev):
                order = lev.argsort(stable=True)
                return order.split(torch.bincount(lev).tolist())
            lev = new

    def ragged(first, last):
        cnt = last - first
        own = torch.repeat_interleave(torch.arange(len(cnt), device=d), cnt)
        return own, torch.arange(len(own), device=d) - (cnt.cumsum(0) - cnt)[own] + first[own]
    inv = torch.zeros(N, 4, 4, dtype=torch.float64, device=d)
    low = levels(col < row)
    for rows in low:
        nl = diag[rows] - ia[rows]
        for t in range(int(nl.max())):
            i = rows[nl > t]
            at = ia[i] + t
            k = col[at]
            A[at] = A[at] @ inv[k]
            own, kj = ragged(diag[k] + 1, ia[k + 1])
            want = i[own] * N + col[kj]
            pos = torch.searchsorted(key, want).clamp_(max=len(key) - 1)
            hit = key[pos] == want
            A[pos[hit]] -= A[at[own[hit]]] @ A[kj[hit]]
        inv[rows] = torch.linalg.inv(A[diag[rows]])
    x = torch.zeros(N, 4, dtype=torch.float64, device=d)
    x[rank] = b
    for sets, upper in ((low, False), (levels(col > row), True)):
        for rows in sets:
            own, j = ragged(*((diag[rows] + 1, ia[rows + 1]) if upper else (ia[rows], diag[rows])))
            t = torch.zeros(len(rows), 4, dtype=torch.float64, device=d)
            t.index_add_(0, own, (A[j] @ x[col[j]][:, :, None])[:, :, 0])
            x[rows] -= t
            if upper:
                x[rows] = (inv[rows] @ x[rows][:, :, None])[:, :, 0]
    return x[rank]


# (outputs, stored inputs, inputs) of the network's linear maps; the bias is the column after the inputs
_MAPS = [(32, 16, 8), (32, 48, 32)] + [(32, 80, 68), (32, 48, 32), (32, 80, 64), (32, 48, 32)] * 3 + [(32, 48, 32), (16, 48, 32)]


def _exact_network(G, theta, x0):
    """The message-passing network on node features x0, all in 64 bits."""
    W, o = [], 0
    for out, kin, real in _MAPS:
        W.append((theta[o:o + out * kin].view(out, kin), real))
        o += out * kin

    def mlp(k, x):
        for j in (k, k + 1):
            w, real = W[j]
            x = x @ w[:, :real].T + w[:, real]
            x = torch.relu(x) if j == k else x
        return x
    i, j = torch.cat([G.n0, G.n1]), torch.cat([G.n1, G.n0])
    a = (G.area / G.area.mean())[:, None]
    feat = torch.cat([torch.cat([G.nrm, a], 1), torch.cat([-G.nrm, a], 1)])
    h = mlp(0, x0)
    for l in range(3):
        m = mlp(2 + 4 * l, torch.cat([h[i], h[j], feat], 1))
        s = torch.zeros_like(h).index_add(0, i, m)
        h = h + mlp(4 + 4 * l, torch.cat([h, s], 1))
    return mlp(14, h)[:, :4]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("solve", "flexible"):
        return None   # an iterate stopped by a tolerance: no value of its own in 64 bits
    m = _mesh(case)
    G = _Geo(m.view)
    aoa, q, rng = _state(case, seed)
    Q = torch.from_numpy(q).to(G.d).view(-1, 4)
    if kind == "residual":
        grad, r = _exact_residual(G, Q, aoa, case["first_order"])
        return {"gx": grad[:, 0].reshape(-1), "gy": grad[:, 1].reshape(-1), "gz": grad[:, 2].reshape(-1), "r": r.reshape(-1)}
    if kind in ("precond", "trisolve"):
        b = torch.from_numpy(rng.standard_normal(q.size)).to(G.d).view(-1, 4)
        if kind == "trisolve":
            aoa, q, _ = _state(case, 0)
            Q = torch.from_numpy(q).to(G.d).view(-1, 4)
        rank = torch.arange(G.N)
        if case["order"] == "spatial":   # the elimination order is part of the plan
            _settings(case, aoa)
            m.flux(q)
            rank = torch.from_numpy(m.ilu_rank())
        cdt = _exact_timestep(G, Q)
        x = _exact_factor_solve(G, Q, aoa, cdt, rank, b).reshape(-1)
        return {"x": x} if kind == "trisolve" else {"cdt": cdt, "x": x}
    theta = torch.from_numpy(_weights().astype(np.float64)).to(G.d)
    y = torch.from_numpy(0.01 * rng.standard_normal(q.size)).to(G.d).view(-1, 4)
    if kind == "network":
        s = y.square().mean().sqrt()
        return {"z": (y + s * _exact_network(G, theta, torch.cat([y / s, Q], 1))).reshape(-1)}
    theta.requires_grad_(True)
    pairs = _pairs(case, q, rng, G.d)
    loss = 0.0
    for x0, t in pairs:
        part = (_exact_network(G, theta, x0.double()) - t.double()).square().sum() / (len(pairs) * 4 * G.N)
        part.backward()
        loss += float(part)
    return {"loss": loss, "grad": theta.grad}
