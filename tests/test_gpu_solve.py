"""The device MINRES against the system it solved, over the forms its kernel
takes: fewer rows than a thread block's, all records in shared memory, records
that stream, vectors in shared memory in full, in part and not at all, a halo
too large for shared memory, and more iterations than one launch runs."""
import numpy as np
import pytest

from icflow_b200 import mesh as M
from icflow_b200.model_prms import config_prms

pytestmark = pytest.mark.gpu


def _context(coll, h, seed=0):
    from icflow_b200.gpu_functionality import GPU_Functionality

    gf = GPU_Functionality(0)
    gf.prms = config_prms(penaltyK=1e8)
    gf.mc = coll
    gf.SetConstants()
    gf.TransferStaticDataToDevice()
    rng = np.random.default_rng(seed)
    n, nc = len(coll.x0), len(coll.czs)
    ext = np.ptp(coll.x0, axis=0).max()
    un = (rng.random((n, 3)) - 0.5) * 1e-6 * ext
    un[coll.anchored] = 0.0
    gf.TransferPCSR(np.zeros((nc, 3)), np.zeros((nc, 3)), np.zeros(nc, np.int32))
    gf.TransferNodesToGPU(un, (rng.random((n, 3)) - 0.5) * 1e-3, rng.random((n, 3)) - 0.5)
    gf.CreateStructure()
    gf.AssembleElemsAndCZs(h)
    return gf


def _system(gf):
    from scipy.sparse import bsr_matrix

    ls = gf.linearSystem
    vals, rhs = gf.TransferLinearSystemToHost()
    U = bsr_matrix((vals.reshape(-1, 3, 3), ls.csr_cols, ls.csr_rows), shape=(3 * ls.N, 3 * ls.N)).tocsr()
    row = np.repeat(np.arange(ls.N), np.diff(ls.csr_rows))
    diag = vals.reshape(-1, 3, 3)[row == ls.csr_cols]
    D = bsr_matrix((diag, np.arange(ls.N), np.arange(ls.N + 1)), shape=U.shape).tocsr()
    return (U + U.T - D).tocsr(), rhs, np.linalg.inv(diag)


def _random_tets(n, seed=0):
    """n nodes at random in a cube, each in about five tets of random nodes: a
    piece of the row order has almost no column in common."""
    rng = np.random.default_rng(seed)
    x0 = rng.random((n, 3))
    el = np.concatenate([rng.permutation(n)[:n - n % 4].reshape(-1, 4) for _ in range(5)])
    flip = M._jdet(x0[el]) < 0
    el[flip] = el[flip][:, [0, 1, 3, 2]]
    m = M.Mesh(x0=x0, elems=el, faces=el[:1, :3], face_exposed=np.ones(1, bool))
    return M.Collection([m]).prepare()


def _box(n):
    return M.Collection([M.box_mesh((n, n, n), (1e-3, 1e-3, 1e-3))]).prepare()


CASES = {
    "one tet": (lambda: M.Collection([M.Mesh(x0=np.array([[0, 0, 0], [1e-3, 0, 0], [0, 1e-3, 0], [0, 0, 1e-3]], float),
                                             elems=np.array([[0, 2, 1, 3]]), faces=np.array([[0, 1, 2]]),
                                             face_exposed=np.ones(1, bool))]).prepare(), 1e-6),
    "beam": (M.cantilever, 1e-4),
    "polycrystal 5": (lambda: M.polycrystal(n=5, grains=3, platens=False), 1e-6),
    "polycrystal 13": (lambda: M.polycrystal(n=13, grains=9, platens=False), 1e-6),
    "polycrystal 27": (lambda: M.polycrystal(n=27, grains=80, platens=False), 1e-6),
    "vectors in part": (lambda: _box(47), 1e-7),   # 110,592 rows
    "vectors in global memory": (lambda: _box(59), 1e-7),   # 216,000 rows
    "no halo": (lambda: _random_tets(84001), 1e-9),
}


@pytest.mark.parametrize("name", list(CASES))
def test_solve_reaches_its_residual(name):
    make, h = CASES[name]
    coll = make()
    if name == "one tet":  # oriented like the generators' meshes
        coll.elems[M._jdet(coll.x0[coll.elems]) < 0] = coll.elems[:, [0, 1, 3, 2]]
    gf = _context(coll, h)
    tol = 1e-10
    it, rel, dx = gf.Solve(tol, want_dx=True)
    again = gf.Solve(tol, want_dx=True)[2]
    assert np.array_equal(dx, again)  # every sum in a fixed order
    A, b, Dinv = _system(gf)
    gf.close()
    norm = lambda r: np.sqrt(np.einsum("ri,rij,rj->", r.reshape(-1, 3), Dinv, r.reshape(-1, 3)))  # noqa: E731
    x = dx.ravel()
    # the recursion's residual may drift from the true one by a rounding of
    # the products per iteration
    drift = it * 2.0 ** -52 * norm(abs(A) @ np.abs(x) + np.abs(b)) / norm(b)
    assert rel <= tol and it % 4 == 0
    assert norm(b - A @ x) / norm(b) <= tol + drift


def test_solve_past_one_launch():
    """2,100 iterations, more than one launch runs: the state carried over
    keeps the solution that the iteration had reached long before."""
    from icflow_b200._lib import ICFError

    gf = _context(M.polycrystal(n=7, grains=4, platens=False), 1e-6)
    _, _, dx = gf.Solve(1e-13, want_dx=True)
    A, b, Dinv = _system(gf)
    n = len(gf.mc.x0)
    gf.SetDU(np.zeros((n, 3)))
    with pytest.raises(ICFError, match="no convergence in 2100"):
        gf.Solve(1e-250, max_iter=2100)
    gf.ApplyDx()
    du = gf.GetNodeState()[3]
    gf.close()
    x = du[gf.mc.alt >= 0].ravel()
    norm = lambda r: np.sqrt(np.einsum("ri,rij,rj->", r.reshape(-1, 3), Dinv, r.reshape(-1, 3)))  # noqa: E731
    drift = 2100 * 2.0 ** -52 * norm(abs(A) @ np.abs(x) + np.abs(b)) / norm(b)
    assert norm(b - A @ x) / norm(b) <= 1e-13 + drift
