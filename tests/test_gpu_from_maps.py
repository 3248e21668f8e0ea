"""Meshes made from maps (DA.from_maps) that no octree gives."""
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def one_octet(faces):
    """The 8 children of one octet (the whole domain, maxDepth 1); the points at the centres of `faces` (axis, side)
    hang although the points on the faces' edges do not."""
    ids, at = {}, []
    hangs = set()
    for axis, side in faces:
        p = [1, 1, 1]
        p[axis] = 2 * side
        hangs.add(tuple(p))
    for p in sorted(itertools.product(range(3), repeat=3), key=lambda p: [(p[2 - k % 3] >> (1 - k // 3)) & 1 for k in range(6)]):
        if p not in hangs:
            ids[p] = len(at)
            at.append(p)
    nl, hm = np.zeros((8, 8), np.uint32), np.zeros(8, np.uint8)
    for c in range(8):
        for v in range(8):
            p = tuple(((c >> a) & 1) + ((v >> a) & 1) for a in range(3))
            if p in hangs:
                hm[c] |= 1 << v
                p = tuple(2 * ((v >> a) & 1) for a in range(3))
            nl[c, v] = ids[p]
    exyz = np.array([[(c >> a) & 1 for a in range(3)] for c in range(8)], np.uint32)
    return dict(max_depth=1, nlist=nl, level=np.full(8, 2), cnum=np.arange(8), hmask=hm, node_xyz=np.array(at),
                elem_xyz=exyz), len(at)


def diagonal(maps, N, coef):
    """The diagonal of the sum over the elements of T^T (a K + b M) T, T the mean over an element's listed slots."""
    k1, m1 = np.array([[.5, -.5], [-.5, .5]]), np.array([[2., 1.], [1., 2.]]) / 3

    def kron3(x, y, z):
        return np.kron(z, np.kron(y, x))

    K = kron3(k1, m1, m1) + kron3(m1, k1, m1) + kron3(m1, m1, k1)
    M = kron3(m1, m1, m1)
    d = np.zeros(N)
    h = 0.5
    for c in range(8):
        T = np.eye(8)
        for v in range(8):
            if (maps["hmask"][c] >> v) & 1:
                T[v] = [(j & ~(v ^ c) & 7) == 0 for j in [s ^ c for s in range(8)]]
                T[v] /= T[v].sum()
        A = T.T @ (coef[c, 0] * h / 2 * K + coef[c, 1] * h ** 3 / 8 * M) @ T
        np.add.at(d, maps["nlist"][c], np.diag(A))
    return d


# a face's centre alone hangs: outside the 18 patterns that octrees have.  Sums of a few dozen FP64 terms
@pytest.mark.parametrize("faces", [[(2, 0)], [(0, 1)], [(2, 0), (1, 1), (0, 0)], [(a, s) for a in range(3) for s in (0, 1)]])
def test_diagonal_of_other_hanging_patterns(gpu, faces):
    import torch
    maps, N = one_octet(faces)
    da = gpu.DA.from_maps(**maps)
    for coef in (None, np.random.default_rng(1).uniform(1, 2, (8, 2))):
        got = gpu.Jacobian2(da, coef).getDiagonal()
        torch.cuda.synchronize()
        want = diagonal(maps, N, np.ones((8, 2)) if coef is None else coef)
        assert np.abs(got.cpu().numpy() - want).max() <= 1e-14 * np.abs(want).max()
