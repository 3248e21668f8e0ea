"""Octree and mesh set-up at the edges of its hash sets, counts and memory pool."""
import threading

import numpy as np
import pytest

from dendro_b200 import inputs as I

pytestmark = pytest.mark.gpu


def same(a, b):
    return len(a) == len(b) and np.array_equal(a.view(np.uint32).reshape(-1, 4), b.view(np.uint32).reshape(-1, 4))


def pairs_at_corners(places, depth):
    """Pairs of points in neighbouring finest cells at corners of a coarse grid: balancing such an octree makes it
    seven times larger, more than the set of internal octants first has room for."""
    c = np.unique(np.round(np.random.default_rng(3).uniform(0.1, 0.9, (places, 3)) * 16) / 16, axis=0)
    return np.concatenate([c + 2.0 ** -(depth + 1), c + 3 * 2.0 ** -(depth + 1)])


def check_mesh(gpu, oracle, pts, depth):
    lin = oracle.points2octree(pts, depth, 1)
    ref = oracle.balance(lin, depth)
    assert same(gpu.points2Octree(pts, depth, 1).to_numpy(), lin)
    bal = gpu.balanceOctree(gpu.Octree.from_octants(lin, depth))
    assert same(bal.to_numpy(), ref)
    m = oracle.Mesh(ref, depth)
    da = gpu.DA(bal)
    got = da.export()
    assert (da.E, da.N) == (m.E, m.N)
    for k, want in (("nlist", m.nlist), ("hmask", m.hmask), ("cnum", m.cnum), ("etype", m.etype), ("level", m.elev),
                    ("node_xyz", m.node_xyz)):
        assert np.array_equal(got[k], want), k


# one octet, one level, tiles of 2048 octants just filled or overrun, a set that is built again
@pytest.mark.parametrize("n,depth", [(2, 1), (2, 2), (9, 3), (330, 6), (700, 5), (3000, 12)])
def test_mesh_sizes(gpu, oracle, n, depth):
    check_mesh(gpu, oracle, I.clamp_unit(I.uniform_cloud(n, n), depth), depth)


def test_mesh_of_a_set_built_again(gpu, oracle):
    pts = pairs_at_corners(64, 17)
    lin = oracle.points2octree(pts, 17, 1)
    assert (len(oracle.balance(lin, 17)) - 1) // 7 > max(4096, 4 * (len(lin) // 7))
    check_mesh(gpu, oracle, pts, 17)


def test_set_up_in_several_threads(gpu, oracle):
    clouds = [I.clamp_unit(I.gaussian_cloud(1500 + 900 * i, i), 9) for i in range(4)]
    refs = [oracle.balance(oracle.points2octree(p, 9, 1), 9) for p in clouds]
    nls = [oracle.Mesh(r, 9).nlist for r in refs]
    bad = []

    def work(i):
        for _ in range(5):
            t = gpu.balanceOctree(gpu.points2Octree(clouds[i], 9, 1))
            if not same(t.to_numpy(), refs[i]) or not np.array_equal(gpu.DA(t).export()["nlist"], nls[i]):
                bad.append(i)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


def test_first_use_of_a_mesh_in_several_threads(gpu):
    """Threads that share a new mesh, each with its own operators and stream, all find its tables built once."""
    import torch
    da = gpu.DA(gpu.balanceOctree(gpu.points2Octree(I.clamp_unit(I.gaussian_cloud(20000, 3), 10), 10, 1)))
    one = gpu.DA(gpu.balanceOctree(gpu.points2Octree(I.clamp_unit(I.gaussian_cloud(20000, 3), 10), 10, 1)))
    x = torch.rand(da.N, dtype=torch.float64, device="cuda")
    x3 = torch.rand(3 * da.N, dtype=torch.float64, device="cuda")
    X = torch.rand(da.N, 64, dtype=torch.float32, device="cuda")

    def forms(d):
        st = torch.cuda.current_stream()
        e, J = gpu.Elasticity(d, 0.4, 0.6), gpu.Jacobian2(d)
        return [J.mult(x, stream=st), e.mult(x3, stream=st), J.mult_multi(X, split=5, stream=st)]

    want = forms(one)
    torch.cuda.synchronize()
    start = threading.Barrier(4)
    got = [None] * 4

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            start.wait()
            got[i] = forms(da)
            torch.cuda.current_stream().synchronize()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for g in got:
        for a, b, tol in zip(g, want, (1e-13, 1e-13, 1e-5)):
            assert (a - b).abs().max() <= tol * b.abs().max()


def test_a_mesh_is_tuned_once_by_threads_that_share_it(gpu):
    """Whichever thread times the launch shapes, all threads run the one that it chose."""
    import torch
    pts = I.clamp_unit(I.gaussian_cloud(4000, 3), 10)
    for _ in range(6):
        da = gpu.DA(gpu.balanceOctree(gpu.points2Octree(pts, 10, 1)))
        x = torch.rand(da.N, dtype=torch.float64, device="cuda")
        names, start = [None] * 4, threading.Barrier(4)

        def work(i):
            st = torch.cuda.Stream()
            J = gpu.Jacobian2(da)
            start.wait()
            J.mult(x, torch.empty_like(x), stream=st)
            names[i] = J.kernel_name()
            st.synchronize()

        threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert names == [gpu.Jacobian2(da).kernel_name()] * 4


def test_first_use_of_a_mesh_inside_a_capture(gpu):
    """A table that a captured call is the first to need is there when the call returns, for the graph and for the
    calls after it."""
    import torch
    pts = I.clamp_unit(I.gaussian_cloud(5000, 3), 10)
    da, one = (gpu.DA(gpu.balanceOctree(gpu.points2Octree(pts, 10, 1))) for _ in range(2))
    X = torch.rand(da.N, 64, dtype=torch.float32, device="cuda")
    want = gpu.Jacobian2(one).mult_multi(X, split=5)
    Y = torch.zeros_like(X)
    A = gpu.Jacobian2(da)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="relaxed"):
        A.mult_multi(X, Y, split=5, stream=torch.cuda.current_stream())
    for _ in range(2):
        Y.fill_(7.0)
        g.replay()
        torch.cuda.synchronize()
        assert (Y - want).abs().max() <= 1e-5 * want.abs().max()
    del g
    Y = A.mult_multi(X, split=5)
    assert (Y - want).abs().max() <= 1e-5 * want.abs().max()


def test_set_up_and_release_beside_a_capture(gpu):
    """A thread that makes, uses and releases octrees, meshes, operators and hierarchies does not end the capture of
    another thread's stream."""
    import torch
    pts = I.clamp_unit(I.gaussian_cloud(3000, 3), 9)
    x = torch.rand(1000, dtype=torch.float64, device="cuda")
    y = torch.zeros_like(x)
    st = torch.cuda.Stream()
    bad = []

    def work():
        try:
            t = gpu.balanceOctree(gpu.points2Octree(pts, 9, 1))
            da = gpu.DA(t)
            A = gpu.Jacobian2(da)
            A.mult(v[0][:da.N], v[1][:da.N], stream=st)
            m = gpu.DAMG(t, nlevels=3)
            m.setKSP()
            m.setKSP(np.full((da.E, 2), 2.0))
            del A, m, da, t
        except Exception as e:  # noqa: BLE001 -- the test's thread reports it
            bad.append(e)

    v = torch.ones((2, 100000), dtype=torch.float64, device="cuda")
    work()  # loads the kernels
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="thread_local"):
        torch.mul(x, 2.0, out=y)
        th = threading.Thread(target=work)
        th.start()
        th.join()
        y.add_(1.0)
    assert not bad
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, 2 * x + 1)


def test_operators_are_ready_on_any_stream(gpu):
    """What creating an operator computes is there when the call returns, although the default stream is busy."""
    import torch
    da = gpu.DA(gpu.balanceOctree(gpu.points2Octree(I.clamp_unit(I.gaussian_cloud(3000, 3), 9), 9, 1)))
    st = torch.cuda.Stream()
    for make in (lambda: gpu.Elasticity(da, 0.4, 0.6), lambda: gpu.DirichletLaplacian(da),
                 lambda: gpu.Jacobian2(da, np.full((da.E, 2), 3.0))):
        A = make()
        x = torch.rand(A.n, dtype=torch.float64, device="cuda")
        want = A.mult(x)
        y = torch.empty_like(x)
        torch.cuda.synchronize()
        del A
        torch.full((da.N + 64 * da.E,), 255, dtype=torch.uint8, device="cuda")  # what new flags may find
        torch.cuda._sleep(100_000_000)
        make().mult(x, y, stream=st)
        st.synchronize()
        assert (y - want).abs().max() <= 1e-13 * want.abs().max()


def test_solves_beside_another_threads_graph(gpu):
    """One thread captures its V-cycle, again after every change of its operator, while others solve: a solve waits
    for the device before it starts, which would end the capture."""
    import torch
    trees = [gpu.balanceOctree(gpu.points2Octree(I.clamp_unit(I.gaussian_cloud(n, n), 11), 11, 1))
             for n in (20000, 50, 60, 70)]
    ms = [gpu.DAMG(t, inner_prec=1, use_graph=i == 0) for i, t in enumerate(trees)]
    for m in ms:
        m.setKSP()
    bs = [torch.rand(int(m.N[0]), dtype=torch.float64, device="cuda") for m in ms]
    for m, b in zip(ms, bs):
        m.solve(b)
    bad, start, done = [], threading.Barrier(4), threading.Event()

    def work(i):
        try:
            start.wait()
            if i == 0:
                for _ in range(30):
                    ms[0].setKSP()
                    ms[0].solve(bs[0])
            while i and not done.is_set():
                ms[i].solve(bs[i])
        except Exception as e:  # noqa: BLE001 -- the test's thread reports it
            bad.append((i, e))
        finally:
            if i == 0:
                done.set()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad


def test_levels_of_a_batch_have_octets(gpu, oracle):
    """Every octet launch shape on a batch's concatenated mesh, against the meshes one by one."""
    import torch
    clouds = [I.clamp_unit(I.gaussian_cloud(n, n), 8) for n in (300, 1700, 40)]
    trees = [gpu.balanceOctree(gpu.points2Octree(p, 8, 1)) for p in clouds]
    m = gpu.DAMG(trees, nlevels=3)
    da = m.level_da(0)
    _, no = m.batch_offsets(0)
    x = np.random.default_rng(0).uniform(-1, 1, da.N)
    want = np.concatenate([oracle.Mesh(t.to_numpy(), 8).matvec(x[no[i]:no[i + 1]]) for i, t in enumerate(trees)])
    A = gpu.Jacobian2(da)
    for v in range(A.kernel_count()):
        A.set_kernel(v)
        y = A.mult(torch.tensor(x, device="cuda")).cpu().numpy()
        assert np.linalg.norm(y - want) <= 1e-12 * np.linalg.norm(want), v


@pytest.fixture
def no_memory(gpu):
    """Calls of this thread find no memory for blocks above the given size."""
    yield gpu.setAllocationLimit
    gpu.setAllocationLimit(0)


# FP64 and FP32 on a mesh timed in L2 and on one timed from HBM
@pytest.mark.parametrize("n,depth", [(3000, 9), (262144, 13)])
def test_operator_without_memory_for_tables(gpu, no_memory, n, depth):
    import torch
    das = [gpu.DA(gpu.balanceOctree(gpu.points2Octree(I.clamp_unit(I.lognormal_cloud(n, 5), depth), depth, 1)))
           for _ in range(2)]
    for dt, tol in ((torch.float64, 1e-13), (torch.float32, 1e-5)):
        x = torch.rand(das[0].N, dtype=dt, device="cuda")
        want = gpu.Jacobian2(das[0]).mult(x)
        no_memory(1)
        y = gpu.Jacobian2(das[1]).mult(x)
        no_memory(0)
        assert (y - want).abs().max() <= tol * want.abs().max()


def test_elasticity_without_memory_for_tiles(gpu, oracle, no_memory):
    import torch
    octs = oracle.balance(oracle.points2octree(I.clamp_unit(I.gaussian_cloud(2000, 5), 9), 9, 1), 9)
    ref, da = oracle.Mesh(octs, 9), gpu.DA(gpu.Octree.from_octants(octs, 9))
    x = np.random.default_rng(2).uniform(-1, 1, 3 * ref.N)
    want = ref.elasticity_matvec(x, 0.4, 0.6, ref.node_bdy)
    no_memory(2 * ref.N)  # the operator's own flags, one byte per node, and no tile table
    few = gpu.Elasticity(da, 0.4, 0.6)
    for A in (few, no_memory(0) or gpu.Elasticity(da, 0.4, 0.6), few):  # with the tiles that the second one builds
        y = A.mult(torch.tensor(x, device="cuda")).cpu().numpy()
        assert np.linalg.norm(y - want) <= 1e-12 * np.linalg.norm(want)


# only the import is called: what it refuses reaches no other kernel
@pytest.mark.parametrize("octants,depth", [([(16, 0, 0, 4), (17, 0, 0, 4)], 4), ([(0, 0, 0, 4), (0, 16, 0, 4)], 4),
                                           ([(0, 0, 0, 1), (0, 0, 1 << 21, 1)], 4), ([(0, 0, 0, 3), (8, 8, 8, 3)], 3),
                                           ([(1, 0, 0, 0)], 0), ([(1 << 19, 0, 0, 19)], 19)])
def test_octants_outside_the_domain_are_refused(gpu, tmp_path, octants, depth):
    from dendro_b200._lib import OCT_DTYPE
    with pytest.raises(gpu.DendroError) as err:
        gpu.Octree.from_octants(np.array(octants, OCT_DTYPE), depth)
    assert err.value.status == 6  # DG_EUNBALANCED
    f = tmp_path / "o.ot"
    f.write_text(f"3 {depth}\n{len(octants)}\n" + "".join("%d %d %d %d\n" % o for o in octants))
    with pytest.raises(gpu.DendroError):
        gpu.readNodesFromFile(f)


@pytest.mark.parametrize("depth", [1, 4, 19])
def test_octants_at_the_far_corner_are_kept(gpu, depth):
    from dendro_b200._lib import OCT_DTYPE
    top = (1 << depth) - 1
    a = np.array([(0, 0, 0, depth), (top, top, top, depth)], OCT_DTYPE)
    assert same(gpu.Octree.from_octants(a, depth).to_numpy(), a)


def test_transfers_of_host_vectors_see_this_call_s_data(gpu):
    """The prolongation keeps constants and the restriction is linear, also where the vector's last part has only just
    been copied."""
    m = gpu.DAMG(gpu.balanceOctree(gpu.points2Octree(I.clamp_unit(I.lognormal_cloud(20000, 3), 12), 12, 1)), nlevels=2)
    nf, nc = int(m.N[0]), int(m.N[1])
    one = m.restrict(0, np.ones(nf))
    for k in range(40):
        c = 1.0 + k
        xf = m.prolong(0, np.full(nc, c), np.zeros(nf))
        assert (np.abs(xf - c) <= 1e-14 * c).all()
        assert (np.abs(m.restrict(0, np.full(nf, c)) - c * one) <= 1e-13 * c * one).all()
