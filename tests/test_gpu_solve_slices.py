"""A solve over several launches of the solver's kernel: the state that a launch
leaves for the next is complete, so that slices of 4 and of 32 iterations give
the solution of a single launch bit for bit, after as many iterations.  Over
the forms that carry the state differently: all vectors in shared memory with
and without streamed records, vectors in part, in global memory, no halo."""
import ctypes as C

import numpy as np
import pytest

from icflow_b200 import _lib
from tests.test_gpu_solve import CASES, M, _context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", list(CASES))
def test_slices_give_the_same_solution(name):
    make, h = CASES[name]
    coll = make()
    if name == "one tet":  # oriented like the generators' meshes
        coll.elems[M._jdet(coll.x0[coll.elems]) < 0] = coll.elems[:, [0, 1, 3, 2]]
    gf = _context(coll, h)
    fn = _lib.load().icf_solver_slice
    fn.argtypes, fn.restype = [C.c_void_p, C.c_int], C.c_int
    assert fn(gf.ctx, 6) != 0 and fn(gf.ctx, -4) != 0
    assert fn(gf.ctx, 8192) == 0
    whole = gf.Solve(1e-10, want_dx=True)
    assert whole[0] <= 8192  # a single launch
    for n in (4, 32, 0):  # (0: as a caller's solves run)
        assert fn(gf.ctx, n) == 0
        it, rel, dx = gf.Solve(1e-10, want_dx=True)
        assert (it, rel) == whole[:2], n
        assert np.array_equal(dx, whole[2]), n
    gf.close()
