"""A contact with a node that no tet or cohesive zone holds joins the rows of its
face to a column without a row.  The structure takes it; the solve, which has no
equation for that node, says so, and the context solves again without it.  An
increment leaves such a node where it is."""
import numpy as np
import pytest

from icflow_b200 import mesh as M
from icflow_b200._lib import ICFError
from icflow_b200.model_prms import config_prms

pytestmark = pytest.mark.gpu


def _context():
    from icflow_b200.gpu_functionality import GPU_Functionality

    x0 = np.array([[0, 0, 0], [1e-3, 0, 0], [0, 1e-3, 0], [0, 0, 1e-3], [3e-4, 3e-4, -1e-4]])
    coll = M.Collection([M.Mesh(x0=x0, elems=np.array([[0, 2, 1, 3]]), faces=np.array([[0, 1, 2]]),
                                face_exposed=np.ones(1, bool))]).prepare()
    coll.elems[M._jdet(coll.x0[coll.elems]) < 0] = coll.elems[:, [0, 1, 3, 2]]
    gf = GPU_Functionality(0)
    gf.prms = config_prms(penaltyK=1e8)
    gf.mc = coll
    gf.SetConstants()
    gf.TransferStaticDataToDevice()
    gf.TransferPCSR(np.zeros((0, 3)), np.zeros((0, 3)), np.zeros(0, np.int32))
    gf.TransferNodesToGPU(np.full((5, 3), 1e-8), np.zeros((5, 3)), np.zeros((5, 3)))
    return gf


def test_column_without_a_row():
    gf = _context()
    out = []
    for imp in ([], [[4, 0, 1, 2]], []):
        gf.SetImpacts(np.array(imp, np.int32).reshape(-1, 4))
        N, nnz = gf.CreateStructure()
        assert (N, nnz) == (4, 10 + 3 * len(imp))
        gf.AssembleElemsAndCZs(1e-6)
        if imp:
            assert gf.linearSystem.csr_cols.max() == 4
            for _ in range(2):
                with pytest.raises(ICFError, match="outside the system"):
                    gf.Solve(1e-10)
        else:
            out.append(gf.Solve(1e-10, want_dx=True)[2])
    gf.close()
    assert np.array_equal(out[0], out[1])


def test_increment_of_a_node_without_a_row():
    gf = _context()
    gf.SetImpacts(np.zeros((0, 4), np.int32))
    gf.CreateStructure()
    gf.AssembleElemsAndCZs(1e-6)
    dx = gf.Solve(1e-10, want_dx=True)[2]
    start = np.arange(15.0).reshape(5, 3)
    for add in (gf.ApplyDx, lambda: gf.XtoDU(dx)):
        gf.SetDU(start)
        add()
        du = gf.GetNodeState()[3]
        assert np.array_equal(du[4], start[4])
        assert np.array_equal(du[:4], start[:4] + dx)
    gf.close()
