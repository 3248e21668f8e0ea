"""The work that a program on this package has it do, as cases to time and compare.

Five kinds, all through the public entry points:

* ``apply``: one application of an operator on a mesh -- the Laplacian + mass operator of
  ``Jacobian2`` on FP64 or FP32 vectors, with unit or per-element coefficients, or
  ``Elasticity`` (3 values per node).  The inner loop of every Krylov method on top of it.
* ``multi``: ``Jacobian2.mult_multi`` on a block of vectors, node-major.
* ``mesh``: points -> ``points2Octree`` -> ``balanceOctree`` -> ``DA`` -> the operator's
  diagonal, what an adaptive code repeats whenever its points have moved.
* ``solve``: ``DAMG.solve`` (V-cycle preconditioned CG to a relative residual of 1e-8), FP64
  or with the FP32 inner cycle from a CUDA graph, for one mesh or for a batch of independent
  meshes, or for elasticity.
* ``solve_multi``: ``DAMG.solve_multi``, a block of right-hand sides on one mesh.

Point clouds are the seeded ones of ``dendro_b200.inputs``; depths and sizes are those of the
benchmark, the tests and the range between them.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import dendro_b200 as dg
from dendro_b200 import inputs

RTOL = 1e-8


def listed():
    return [
        # the smallest calls: a test-sized mesh (a coarse level, a small part of a partitioned mesh), where a
        # launch's latency is what counts
        dict(name="apply_gauss4k", kind="apply", cloud="gauss", n=4000, depth=9, dtype="f64", coef=False, dof=1),
        # the FP32 operator of mixed-precision programs on a mesh that fits in L2
        dict(name="apply32_gauss131k", kind="apply", cloud="gauss", n=131072, depth=10, dtype="f32", coef=True, dof=1),
        # the benchmark's operator: 1M log-normal points, variable coefficients
        dict(name="apply_lognormal1m", kind="apply", cloud="lognormal", n=1048576, depth=14, dtype="f64", coef=True,
             dof=1),
        # 3-dof elasticity on the same kind of mesh
        dict(name="elasticity_lognormal1m", kind="apply", cloud="lognormal", n=1048576, depth=14, dtype="f64",
             coef=False, dof=3),
        # many right-hand sides at once, the entry point's default precision
        dict(name="multi64_uniform512k", kind="multi", cloud="uniform", n=524288, depth=12, nrhs=64, split=3,
             coef=False),
        # mesh set-up from points: an ordinary size and the largest
        dict(name="mesh_gauss131k", kind="mesh", cloud="gauss", n=131072, depth=10, maxpts=1),
        dict(name="mesh_lognormal1m", kind="mesh", cloud="lognormal", n=1048576, depth=14, maxpts=1),
        # the plain FP64 solve with 4 levels (a coarsest level of about 18K nodes)
        dict(name="solve_gauss131k", kind="solve", cloud="gauss", n=131072, depth=10, nlevels=4, prec=0, graph=False,
             coef=False, dof=1, count=1),
        # the mixed-precision solve of a large variable-coefficient problem
        dict(name="solve32_lognormal1m", kind="solve", cloud="lognormal", n=1048576, depth=14, nlevels=30, prec=1,
             graph=True, coef=True, dof=1, count=1),
        # elasticity multigrid, an odd size
        dict(name="solve_elasticity_lognormal77k", kind="solve", cloud="lognormal", n=77777, depth=12, nlevels=30,
             prec=0, graph=False, coef=False, dof=3, count=1),
        # independent meshes of uneven sizes solved as one batch
        dict(name="solve_batch8_gauss", kind="solve", cloud="gauss", n=30000, depth=12, nlevels=30, prec=1, graph=True,
             coef=False, dof=1, count=8),
        # a block of right-hand sides solved together
        dict(name="solve_multi32_uniform60k", kind="solve_multi", cloud="uniform", n=60001, depth=11, nlevels=30,
             prec=1, nrhs=32),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["apply", "apply", "elasticity", "multi", "mesh", "solve", "solve", "solve_elasticity", "batch",
                       "solve_multi"])
    cloud = rng.choice(["gauss", "lognormal", "uniform"])
    # the depth that the benchmark gives clouds of this kind, or one less or more
    depth = {"gauss": 11, "lognormal": 13, "uniform": 11}[cloud] + rng.choice([-1, 0, 1])
    if kind == "apply":
        return dict(kind="apply", cloud=cloud, n=_log(rng, 1000, 1000000), depth=depth,
                    dtype=rng.choice(["f64", "f64", "f32"]), coef=rng.random() < 0.5, dof=1)
    if kind == "elasticity":
        return dict(kind="apply", cloud=cloud, n=_log(rng, 1000, 600000), depth=depth, dtype="f64", coef=False, dof=3)
    if kind == "multi":
        split = rng.choice([3, 3, 0, 1])
        nrhs = rng.choice([32, 64, 96, 128] if split == 0 else [16, 32, 48, 64, 96])
        return dict(kind="multi", cloud=cloud, n=_log(rng, 2000, 200000), depth=depth, nrhs=nrhs, split=split,
                    coef=rng.random() < 0.5)
    if kind == "mesh":
        return dict(kind="mesh", cloud=cloud, n=_log(rng, 1000, 800000), depth=depth, maxpts=rng.choice([1, 1, 2, 5]))
    if kind == "solve":
        return dict(kind="solve", cloud=cloud, n=_log(rng, 2000, 400000), depth=depth, nlevels=30,
                    prec=rng.choice([0, 1, 1, 2]), graph=rng.random() < 0.7, coef=rng.random() < 0.5, dof=1, count=1)
    if kind == "solve_elasticity":
        return dict(kind="solve", cloud=cloud, n=_log(rng, 2000, 60000), depth=depth, nlevels=30, prec=0, graph=False,
                    coef=False, dof=3, count=1)
    if kind == "batch":
        return dict(kind="solve", cloud="gauss", n=_log(rng, 2000, 30000), depth=depth, nlevels=30,
                    prec=rng.choice([0, 1]), graph=rng.random() < 0.7, coef=False, dof=1, count=rng.randint(2, 8))
    return dict(kind="solve_multi", cloud=cloud, n=_log(rng, 2000, 60000), depth=depth, nlevels=30,
                prec=rng.choice([0, 1]), nrhs=rng.choice([32, 64]))


def _cloud(cloud, n, depth, number=0):
    if cloud == "gauss":
        p = inputs.gaussian_cloud(n, 7000 + number)
    elif cloud == "lognormal":
        p = inputs.lognormal_cloud(n, 8000 + number)
    else:
        p = inputs.uniform_cloud(n, 9000 + number)
    return inputs.clamp_unit(p, depth)


def _moved(p, depth, seed):
    """Other points of the same cloud: axes permuted and mirrored, every point moved within its finest cell, the
    order shuffled -- another octree of as many octants and nodes, so that outputs of all seeds have one shape."""
    rng = np.random.default_rng([seed, 17])
    side = 1 << depth
    q = np.floor(p * side)[:, rng.permutation(3)]
    mirror = rng.integers(0, 2, 3).astype(bool)
    q[:, mirror] = side - 1 - q[:, mirror]
    return ((q + rng.uniform(0.0, 0.999, q.shape)) / side)[rng.permutation(len(q))]


def _points(case, seed):
    return _moved(_cloud(case["cloud"], case["n"], case["depth"]), case["depth"], seed)


def _octree(case, seed):
    return dg.balanceOctree(dg.points2Octree(_points(case, seed), case["depth"], 1))


def _octrees(case, seed):
    """The balanced octrees of a solve: one, or a batch of uneven sizes (1/4 to 4 times n, around drawn centres)."""
    if case["count"] == 1:
        return [_octree(case, seed)]
    out = []
    for i in range(case["count"]):
        rng = np.random.default_rng([case["n"], i])
        n = max(8, int(round(case["n"] * math.exp(rng.uniform(-math.log(4.0), math.log(4.0))))))
        p = inputs.clamp_unit(rng.normal(rng.uniform(0.3, 0.7, 3), rng.uniform(0.05, 0.2), (n, 3)), case["depth"])
        p = _moved(p, case["depth"], seed * 64 + i)
        out.append(dg.balanceOctree(dg.points2Octree(p, case["depth"], 1)))
    return out


def _rhs(shape, seed, dtype=torch.float64):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.rand(shape, generator=g, dtype=torch.float64, device="cuda") * 2 - 1).to(dtype)


def _coef(case, da):
    return inputs.sphere_coefficients(da.elementCenters()) if case.get("coef") else None


def prepare(case, seed):
    kind = case["kind"]
    if kind == "mesh":
        return dict(case=case, points=torch.tensor(_points(case, seed), device="cuda"))
    if kind in ("apply", "multi"):
        da = dg.DA(_octree(case, seed))
        if kind == "multi":
            x = _rhs((da.N, case["nrhs"]), seed, torch.float32)
            return dict(case=case, da=da, A=dg.Jacobian2(da, _coef(case, da)), x=x, y=torch.empty_like(x))
        if case["dof"] == 3:
            A = dg.Elasticity(da, 1.0 / 2.6, 0.3 / (1.3 * 0.4))  # E = 1, nu = 0.3
        else:
            A = dg.Jacobian2(da, _coef(case, da))
        x = _rhs(case["dof"] * da.N, seed, torch.float64 if case["dtype"] == "f64" else torch.float32)
        return dict(case=case, da=da, A=A, x=x, y=torch.empty_like(x))
    if kind == "solve":
        octs = _octrees(case, seed)
        m = dg.DAMG(octs if case["count"] > 1 else octs[0], nlevels=case["nlevels"], rtol=RTOL,
                    inner_prec=case["prec"], use_graph=case["graph"], dof=case["dof"],
                    **(dict(mu=1.0 / 2.6, lam=0.3 / (1.3 * 0.4)) if case["dof"] == 3 else {}))
        if case["coef"]:
            m.setKSP(_coef(case, m.level_da(0)))
        b = _rhs(case["dof"] * int(m.N[0]), seed)
        return dict(case=case, m=m, b=b, x=torch.empty_like(b))
    m = dg.DAMG(_octree(case, seed), nlevels=case["nlevels"], rtol=RTOL, inner_prec=case["prec"])
    b = _rhs((int(m.N[0]), case["nrhs"]), seed)
    return dict(case=case, m=m, b=b, x=torch.empty_like(b))


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "apply":
        return state["A"].mult(state["x"], state["y"])
    if kind == "multi":
        return state["A"].mult_multi(state["x"], state["y"], split=case["split"])
    if kind == "mesh":
        oct_ = dg.balanceOctree(dg.points2Octree(state["points"], case["depth"], case["maxpts"]))
        da = dg.DA(oct_)
        return dict(octants=len(oct_), nodes=da.N, diagonal=dg.Jacobian2(da).getDiagonal())
    if kind == "solve":
        return state["m"].solve(state["b"], state["x"])[0]
    return state["m"].solve_multi(state["b"], state["x"])[0]


@functools.lru_cache(maxsize=None)
def _sizes(kind, cloud, n, depth, count):
    case = dict(kind=kind, cloud=cloud, n=n, depth=depth, count=count)
    das = [dg.DA(t) for t in (_octrees(case, 1) if kind == "solve" else [_octree(case, 1)])]
    return sum(d.E for d in das), sum(d.N for d in das)


def work(case):
    """Per element its 8 node ids and one word (36 bytes) and its coefficients, per node the vectors' values read
    and written; the element operator in the form with the fewest operations (two 8-point Walsh transforms and 8
    products).  A solve counts 6 iterations of one operator application and a V(2,2) cycle's 4 on every level
    (levels shrink 8-fold) -- the iterations it cannot do without at this tolerance."""
    kind = case["kind"]
    E, N = _sizes(kind, case["cloud"], case["n"], case["depth"], case.get("count", 1))
    if kind == "mesh":
        # points and octants once, the element and node tables written once
        return dict(bytes=24 * case["n"] + 8 * E + 44 * E + 8 * N + 8 * N, flops=8 * 4 * E)
    if kind == "multi":
        return dict(bytes=36 * E + (8 * E if case["coef"] else 0) + 8 * case["nrhs"] * N, flops=56 * case["nrhs"] * E)
    if kind == "apply":
        w = 8 if case["dtype"] == "f64" else 4
        d = case["dof"]
        return dict(bytes=36 * E + (2 * w * E if case["coef"] else 0) + 2 * w * d * N, flops=(56 if d == 1 else 400) * E)
    if kind == "solve":
        w = 8 if case["prec"] == 0 else 4
        d = case["dof"]
        op = 36 * E + (2 * w * E if case["coef"] else 0) + 2 * w * d * N
        return dict(bytes=6 * (1 + 4 * 8 / 7) * op, flops=6 * (1 + 4 * 8 / 7) * (56 if d == 1 else 400) * E)
    w = 8 if case["prec"] == 0 else 4
    op = 36 * E + 2 * w * case["nrhs"] * N
    return dict(bytes=6 * (1 + 4 * 8 / 7) * op, flops=6 * (1 + 4 * 8 / 7) * 56 * case["nrhs"] * E)


# ---- the same in 64 bits with plain torch, from the mesh's maps ----


def _element_matrices(dof, mu=0.0, lam=0.0):
    """Matrices on [-1, 1]^3 that h/2 and h^3/8 scale: (K, M) for dof 1, (mu K (x) I + (mu + lam) GD, None) for 3."""
    k1 = np.array([[1.0, -1.0], [-1.0, 1.0]]) / 2
    m1 = np.array([[2.0, 1.0], [1.0, 2.0]]) / 3
    d1 = np.array([[-1.0, -1.0], [1.0, 1.0]]) / 2  # integral of phi_i' phi_j

    def kron3(x, y, z):  # vertex v = x + 2 y + 4 z
        return np.kron(z, np.kron(y, x))

    K = kron3(k1, m1, m1) + kron3(m1, k1, m1) + kron3(m1, m1, k1)
    if dof == 1:
        return K, kron3(m1, m1, m1)
    G = np.zeros((8, 3, 8, 3))
    for a in range(3):
        for b in range(3):
            f = [m1, m1, m1]
            if a == b:
                f[a] = k1
            else:
                f[a], f[b] = d1, d1.T
            G[:, a, :, b] = (mu + lam) * kron3(*f)
            if a == b:
                G[:, a, :, b] += mu * K
    return G.reshape(24, 24), None


def _groups(da, coef, dof, mu=0.0, lam=0.0):
    """Per child number and hanging mask: its elements' node ids [n, 8], their two scales and the two matrices."""
    m = da.export()
    dev = "cuda"
    nl = torch.from_numpy(m["nlist"].astype(np.int64)).to(dev)
    key = torch.from_numpy(m["cnum"].astype(np.int64) * 256 + m["hmask"]).to(dev)
    h = torch.from_numpy(np.ldexp(1.0, 1 - m["level"].astype(np.int32))).to(dev)
    f1, f2 = h / 2, h ** 3 / 8
    if coef is not None:
        c = torch.from_numpy(np.asarray(coef, np.float64).reshape(-1, 2)).to(dev)
        f1, f2 = f1 * c[:, 0], f2 * c[:, 1]
    K, M = _element_matrices(dof, mu, lam)
    for k in torch.unique(key).tolist():
        idx = torch.nonzero(key == k).reshape(-1)
        cnum, mask = k >> 8, k & 255
        T = np.eye(8)
        for v in range(8):  # a hanging vertex takes the mean of its edge's or face's corners
            if (mask >> v) & 1:
                mid = v ^ cnum
                T[v] = 0
                subs = [s for s in range(8) if s & mid == s]
                for s in subs:
                    T[v, v ^ s] += 1.0 / len(subs)
        if dof == 3:
            T = np.kron(T, np.eye(3))
        mats = [None if A is None else torch.from_numpy(T.T @ A @ T).to(dev) for A in (K, M)]
        yield nl[idx], f1[idx], f2[idx], mats


def _dofs(ids, dof):
    return ids if dof == 1 else (ids[:, :, None] * 3 + torch.arange(3, device=ids.device)).reshape(len(ids), 24)


def _apply64(da, coef, dof, x, **lame):
    """A x for x [n] or [n, columns]."""
    x2 = x.double().reshape(x.shape[0], -1)
    free = None
    if dof == 3:
        free = torch.from_numpy(np.repeat(da.export()["node_bdy"] == 0, 3)).cuda()[:, None]
        src = torch.where(free, x2, torch.zeros_like(x2))
    else:
        src = x2
    y = torch.zeros_like(x2)
    for ids, f1, f2, (K, M) in _groups(da, coef, dof, **lame):
        d = _dofs(ids, dof)
        for c0 in range(0, x2.shape[1], 16):
            u = src[:, c0:c0 + 16][d]  # [n, 8 dof, columns]
            r = f1[:, None, None] * torch.einsum("ij,njc->nic", K, u)
            if M is not None:
                r += f2[:, None, None] * torch.einsum("ij,njc->nic", M, u)
            y[:, c0:c0 + 16].index_add_(0, d.reshape(-1), r.reshape(-1, r.shape[2]))
    if free is not None:
        y = torch.where(free, y, x2)
    return y.reshape(x.shape)


def _csr64(da, coef, dof, **lame):
    n = dof * da.N
    acc_i, acc_v = [], []
    for ids, f1, f2, (K, M) in _groups(da, coef, dof, **lame):
        d = _dofs(ids, dof)
        v = f1[:, None, None] * K
        if M is not None:
            v = v + f2[:, None, None] * M
        acc_i.append((d[:, :, None] * n + d[:, None, :]).reshape(-1))
        acc_v.append(v.reshape(-1))
    i, v = torch.cat(acc_i), torch.cat(acc_v)
    del acc_i, acc_v
    if dof == 3:
        bdy = torch.from_numpy(np.repeat(da.export()["node_bdy"] != 0, 3)).cuda()
        keep = ~(bdy[i // n] | bdy[i % n])
        on = torch.nonzero(bdy).reshape(-1)
        i = torch.cat([i[keep], on * (n + 1)])
        v = torch.cat([v[keep], torch.ones(len(on), dtype=v.dtype, device=v.device)])
    u, inv = torch.unique(i, return_inverse=True)
    w = torch.zeros(len(u), dtype=v.dtype, device=v.device).index_add_(0, inv, v)
    del i, v, inv
    row = u // n
    ptr = torch.searchsorted(row, torch.arange(n + 1, device=u.device))
    A = torch.sparse_csr_tensor(ptr, u % n, w, (n, n))
    diag = torch.zeros(n, dtype=w.dtype, device=w.device)
    on = row == u % n
    diag[row[on]] = w[on]
    return A, diag


def _cg64(A, diag, b, tol=1e-14, maxit=6000):
    """Jacobi-preconditioned CG per column of b [n, columns]; None when it does not get there."""
    x = torch.zeros_like(b)
    r = b.clone()
    z = r / diag[:, None]
    p = z.clone()
    rz = (r * z).sum(0)
    bn = b.norm(dim=0)
    for it in range(maxit):
        q = A @ p
        a = rz / (p * q).sum(0)
        x += a * p
        r -= a * q
        if it % 50 == 49 and bool((r.norm(dim=0) <= tol * bn).all()):
            return x
        z = r / diag[:, None]
        rn = (r * z).sum(0)
        p = z + (rn / rz) * p
        rz = rn
    return None


def exact(case, seed):
    kind = case["kind"]
    lame = dict(mu=1.0 / 2.6, lam=0.3 / (1.3 * 0.4)) if case.get("dof") == 3 else {}
    if kind == "mesh":
        return None  # whole numbers and exact sums of powers of two apart, set-up computes nothing
    if kind in ("apply", "multi"):
        s = prepare(case, seed)
        return _apply64(s["da"], _coef(case, s["da"]), case.get("dof", 1), s["x"], **lame)
    if case["n"] * case.get("count", 1) > 300000:
        return None  # minutes of plain CG
    s = prepare(case, seed)
    octs = _octrees(case, seed) if kind == "solve" else [_octree(case, seed)]
    out, at = [], 0
    for t in octs:
        da = dg.DA(t)
        n = case.get("dof", 1) * da.N
        A, diag = _csr64(da, _coef(case, da), case.get("dof", 1), **lame)
        b = s["b"][at:at + n]
        x = _cg64(A, diag, b.reshape(n, -1))
        if x is None:
            return None
        out.append(x.reshape(b.shape))
        at += n
    return torch.cat(out)
