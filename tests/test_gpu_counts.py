"""The counters of an assembly start from zero on every path and in any order of
paths: the captured graph, direct launches, the profiled launches, the repeat
after new constants."""
import numpy as np
import pytest

from icflow_b200 import _lib
from icflow_b200 import mesh as M
from icflow_b200.model_prms import config_prms
from tests.harness import gpu_assemble, random_state

pytestmark = pytest.mark.gpu


def _values(c):
    return tuple(getattr(c, f) for f, _ in c._fields_)


def test_counts_on_every_path():
    from icflow_b200.gpu_functionality import GPU_Functionality

    coll = M.polycrystal(n=6, grains=5, seed=4, platens=True, gap=-0.3)
    gf = GPU_Functionality(0)
    gf.prms = config_prms(penaltyK=1e8)
    gf.mc = coll
    gf.SetConstants()
    gf.TransferStaticDataToDevice()
    nc = len(coll.czs)
    state = random_state(coll, 3, du=4e-6)
    pairs = M.candidate_pairs(coll, coll.x0 + state[0])
    zero = np.zeros((nc, 3))
    first = _values(gpu_assemble(gf, coll, state, 1e-4, zero, zero, np.zeros(nc, np.int32), pairs=pairs)["counts"])
    assert sum(first[2:]) > 0
    lib = _lib.load()
    for step in ("graph", "graph", "direct", "direct", "profile", "graph", "constants", "graph"):
        if step == "profile":
            gf.ProfileAssembly(1e-4, reps=2)
            continue
        if step == "constants":
            gf.SetConstants()
        _lib.check(gf.ctx, lib.icf_set_graph(gf.ctx, 0 if step == "direct" else 1))
        assert _values(gf.AssembleElemsAndCZs(1e-4)) == first, step
    gf.close()
