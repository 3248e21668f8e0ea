"""Operator kernels at the edges of their tiles and column blocks, against the oracle."""
import numpy as np
import pytest

from dendro_b200 import inputs as I

pytestmark = pytest.mark.gpu


def meshes(gpu, oracle, n, depth, cloud=I.uniform_cloud):
    octs = oracle.balance(oracle.points2octree(I.clamp_unit(cloud(n, n), depth), depth, 1), depth)
    return oracle.Mesh(octs, depth), gpu.DA(gpu.Octree.from_octants(octs, depth))


# FP64 sums of at most a few hundred products each: 1e-12 as for the other operators.  One octet, some, whole
# tiles of 32 octets and a few more (the octet counts of these clouds lie on both sides of 32, 64 and 256)
@pytest.mark.parametrize("n,depth", [(1, 3), (2, 1), (3, 3), (20, 4), (28, 4), (60, 4), (64, 5), (230, 6), (2000, 9)])
@pytest.mark.parametrize("bdy", ["domain", "none", "some", "all"])
def test_elasticity_tiles(gpu, oracle, n, depth, bdy):
    import torch
    ref, da = meshes(gpu, oracle, n, depth)
    rng = np.random.default_rng(n)
    flags = {"domain": ref.node_bdy, "none": np.zeros(ref.N, np.uint8), "all": np.ones(ref.N, np.uint8),
             "some": (rng.random(ref.N) < 0.3).astype(np.uint8)}[bdy]
    x = rng.uniform(-1, 1, 3 * ref.N)
    want = ref.elasticity_matvec(x, 0.4, 0.6, flags)
    A = gpu.Elasticity(da, 0.4, 0.6, None if bdy == "domain" else flags)
    for _ in range(2):  # the second call finds the first one's y
        y = A.mult(torch.tensor(x, device="cuda"), torch.full((3 * ref.N,), 7.0, dtype=torch.float64, device="cuda"))
    assert np.linalg.norm(y.cpu().numpy() - want) <= 1e-12 * np.linalg.norm(want)


# blocks of 64, 32 and 16 columns in every combination; 2e-6: FP32 products and sums of a few dozen terms
@pytest.mark.parametrize("nrhs", [16, 32, 48, 64, 80, 96, 112, 144])
def test_multi_column_blocks(gpu, oracle, nrhs):
    import torch
    ref, da = meshes(gpu, oracle, 700, 7, I.gaussian_cloud)
    c = I.sphere_coefficients(da.elementCenters())
    X = np.random.default_rng(nrhs).uniform(-1, 1, (ref.N, nrhs))
    want = np.stack([ref.matvec(X[:, j], c) for j in range(nrhs)], 1)
    A = gpu.Jacobian2(da, c)
    Xd = torch.tensor(X, dtype=torch.float32, device="cuda")
    for split in (3, 1) + ((0,) if nrhs % 32 == 0 else ()):
        Y = A.mult_multi(Xd, split=split).double().cpu().numpy()
        assert (np.linalg.norm(Y - want, axis=0) / np.linalg.norm(want, axis=0)).max() < 2e-6, split


def test_infinity_stays_in_its_elements(gpu, oracle):
    """An infinite value reaches the nodes of the elements that list its node and no others, in FP32 and FP64, in
    every octet launch shape and with many right-hand sides (an absent child of an octet has no share)."""
    import torch
    ref, da = meshes(gpu, oracle, 400, 7, I.gaussian_cloud)
    x = np.random.default_rng(1).uniform(-1, 1, ref.N)
    at = int(ref.nlist[ref.nlist.shape[0] // 2, 3])
    x[at] = np.inf
    reach = np.zeros(ref.N, bool)
    reach[ref.nlist[(ref.nlist == at).any(1)].reshape(-1)] = True
    A = gpu.Jacobian2(da)
    for v in range(A.kernel_count()):
        for prec, dt in ((0, torch.float64), (1, torch.float32)):
            A.set_kernel(v, prec)
            y = A.mult(torch.tensor(x, dtype=dt, device="cuda")).cpu().numpy()
            assert np.isfinite(y[~reach]).all(), (v, prec)
    X = torch.tensor(np.repeat(x[:, None], 112, 1), dtype=torch.float32, device="cuda")
    Y = A.mult_multi(X).cpu().numpy()
    assert np.isfinite(Y[~reach]).all()


# with 3 values per node (3 x 1874 rows), also after a second set-up: the full inverse has been given back by then
def test_large_dense_coarse_solve_of_elasticity(gpu):
    import torch
    from dendro_b200._lib import check, lib, ptr
    tree = gpu.balanceOctree(gpu.points2Octree(I.clamp_unit(I.gaussian_cloud(250, 7), 7), 7, 1))
    m = gpu.DAMG(tree, nlevels=1, dof=3, mu=0.4, lam=0.2)
    da = m.level_da(0)
    assert 3 * da.N >= 3000
    b = torch.from_numpy(np.random.default_rng(7).uniform(-1, 1, 3 * da.N)).cuda()
    x = torch.empty_like(b)
    for _ in range(2):
        m.setKSP()
        check(lib().dg_damg_coarse_solve(m.h, ptr(b), ptr(x), None), "damg_coarse_solve")
        r = b - gpu.Elasticity(da, 0.4, 0.2).mult(x)
        torch.cuda.synchronize()
        assert float(r.norm() / b.norm()) < 1e-9  # as below


# the packed triangle of a large dense inverse: strips of 16 rows, blocks of 32 columns, the last ones cut short
# (3115, 4071, 5728 and 5244 nodes)
@pytest.mark.parametrize("n", [600, 900, 1200, 1300])
def test_large_dense_coarse_solve(gpu, n):
    import torch
    from dendro_b200._lib import check, lib, ptr
    tree = gpu.balanceOctree(gpu.points2Octree(I.clamp_unit(I.gaussian_cloud(n, n), 8), 8, 1))
    m = gpu.DAMG(tree, nlevels=1)
    m.setKSP()
    da = m.level_da(0)
    assert da.N >= 3000
    b = torch.from_numpy(np.random.default_rng(n).uniform(-1, 1, da.N)).cuda()
    x = torch.empty_like(b)
    check(lib().dg_damg_coarse_solve(m.h, ptr(b), ptr(x), None), "damg_coarse_solve")
    r = b - gpu.Jacobian2(da).mult(x)
    torch.cuda.synchronize()
    assert float(r.norm() / b.norm()) < 1e-9  # rounding times the matrix's condition (h from 1 to 1/256)
