"""The cohesive zones of large models, one lane each, at the edges of a warp and
of a block of lanes: the assembled system, flags, histories and tractions against
the oracle; in mixed precision against the kernel of small models."""
import numpy as np
import pytest

from icflow_b200 import mesh as M
from icflow_b200.model_prms import config_prms
from tests.harness import Oracle, compare, gpu_assemble, oracle_assemble, orc_prms_from, random_state, rowwise_rel

pytestmark = pytest.mark.gpu

LANE, GP = 3, 1  # the variants' indexes
# A mixed block is a sum of three products of FP32 tangents, each of some twenty
# rounded operations: two evaluations differ by at most about 20 x 2^-24.
MIXED_TOL = 20 * 2.0 ** -24


def _context(coll, prms, mixed):
    from icflow_b200.gpu_functionality import GPU_Functionality

    gf = GPU_Functionality(0)
    gf.prms = prms
    gf.mc = coll
    gf.SetPrecision(1 if mixed else 0)
    gf.SetConstants()
    gf.TransferStaticDataToDevice()
    return gf


def _state(coll):
    """Openings from contact over softening to separation; some damaged, some failed."""
    rng = np.random.default_rng(7)
    nc = len(coll.czs)
    pmax = rng.random((nc, 3)) * 2e-6 * (rng.random((nc, 1)) < 0.5)
    failed = (rng.random(nc) < 0.1).astype(np.int32)
    return random_state(coll, 3, du=4e-6), pmax, pmax[:, ::-1].copy(), failed


@pytest.mark.parametrize("nc", [1, 31, 32, 33, 127, 128, 129, 385])
def test_lane_per_cohesive_zone(nc):
    coll = M.polycrystal(n=8, grains=9, seed=0)
    coll.czs = coll.czs[:nc].copy()
    prms = config_prms(penaltyK=1e8)
    O = Oracle()
    state, pmax, tmax, failed = _state(coll)
    none = np.zeros((0, 4), np.int32)
    gf = _context(coll, prms, False)
    gf.SetVariant(4, LANE)
    g = gpu_assemble(gf, coll, state, 1e-4, pmax, tmax, failed, impacts=none)
    gf.close()
    o = oracle_assemble(O, orc_prms_from(O, prms), coll, state, 1e-4, pmax, tmax, none, cz_live=failed == 0)
    compare(g, o)
    out = {}
    for v in (LANE, GP):
        gf = _context(coll, prms, True)
        gf.SetVariant(4, v)
        out[v] = gpu_assemble(gf, coll, state, 1e-4, pmax, tmax, failed, impacts=none)
        gf.close()
    a, b = out[LANE], out[GP]
    assert np.array_equal(a["flags"], b["flags"]) and np.array_equal(a["tent"], b["tent"])
    assert rowwise_rel(b["rows"], b["vals"], a["vals"]) <= MIXED_TOL
    assert np.max(np.abs(a["rhs"] - b["rhs"])) <= 1e-13 * np.max(np.abs(b["rhs"]))
