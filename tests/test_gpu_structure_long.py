"""Contact lists with rows longer than a warp sorts: on both sides of the limit
and far beyond it, between short lists, against the oracle; and such a list costs
no more than some times a list of as many contacts spread over the model."""
import time

import numpy as np
import pytest

from icflow_b200 import mesh as M
from icflow_b200.model_prms import config_prms
from tests.harness import Oracle, compare, gpu_assemble, oracle_assemble, orc_prms_from, random_state

pytestmark = pytest.mark.gpu

ROW_MAX = 512  # codes of a row that a warp sorts


def _longest(coll, imp):
    """Codes of the longest row: pairs of active vertices, the second not before the first."""
    al = coll.alt[imp]
    n = ((al[:, :, None] >= 0) & (al[:, None, :] >= al[:, :, None])).sum(axis=2)
    return int(np.bincount(al[al >= 0], n[al >= 0]).max()) if len(imp) else 0


def _contacts(coll, kind, n, rng):
    free = np.nonzero(coll.alt >= 0)[0]
    faces = coll.faces[rng.integers(0, len(coll.faces), 4 * n + 64)]
    nodes = rng.integers(0, len(coll.x0), len(faces))
    if kind == "last row":  # one code of its row for each contact
        nodes[:] = free[np.argmax(coll.alt[free])]
    elif kind == "one node":
        nodes[:] = free[len(free) // 2]
    elif kind == "one face":
        active = coll.faces[(coll.alt[coll.faces] >= 0).all(axis=1)]
        faces[:] = active[len(active) // 2]
    elif kind == "one contact":
        active = coll.faces[(coll.alt[coll.faces] >= 0).all(axis=1)]
        faces[:], nodes[:] = active[0], free[~np.isin(free, active[0])][-1]
    imp = np.concatenate([nodes[:, None], faces], axis=1)[~(faces == nodes[:, None]).any(axis=1)]
    return imp[:n].astype(np.int32)


LISTS = [("any", 900), ("last row", ROW_MAX - 1), ("last row", ROW_MAX), ("last row", ROW_MAX + 1), ("any", 5),
         ("one contact", 128), ("one contact", 129), ("one face", 2500), ("one node", 6000), ("any", 0),
         ("one face", 20000), ("any", 5000)]


def _context(coll, prms):
    from icflow_b200.gpu_functionality import GPU_Functionality

    gf = GPU_Functionality(0)
    gf.prms = prms
    gf.mc = coll
    gf.SetConstants()
    gf.TransferStaticDataToDevice()
    return gf


def test_long_rows_against_the_oracle():
    coll = M.cantilever()
    O = Oracle()
    prms = config_prms(penaltyK=1e8)
    gf = _context(coll, prms)
    nc = len(coll.czs)
    state = random_state(coll, 0, du=2e-6)
    zero = np.zeros((nc, 3))
    rng = np.random.default_rng(5)
    seen = set()
    for kind, n in LISTS:
        imp = _contacts(coll, kind, n, rng)
        assert len(imp) == n
        seen.add(_longest(coll, imp))
        g = gpu_assemble(gf, coll, state, 1e-4, zero, zero, np.zeros(nc, np.int32), impacts=imp)
        o = oracle_assemble(O, orc_prms_from(O, prms), coll, state, 1e-4, zero, zero, imp)
        compare(g, o)
    gf.close()
    assert {ROW_MAX, ROW_MAX + 1} <= seen and max(seen) > 20 * ROW_MAX


def test_a_long_row_costs_no_more_than_some_lists():
    coll = M.polycrystal(n=12, grains=9, seed=0)
    gf = _context(coll, config_prms(penaltyK=1e8))
    nc = len(coll.czs)
    gf.TransferPCSR(np.zeros((nc, 3)), np.zeros((nc, 3)), np.zeros(nc, np.int32))
    gf.TransferNodesToGPU(*random_state(coll, 0, du=2e-6))
    rng = np.random.default_rng(1)

    def cost(kind):
        lists = [_contacts(coll, kind, 20000, rng) for _ in range(2)]
        best = np.inf
        for k in range(8):  # two lists in turn: each call builds
            gf.SetImpacts(lists[k % 2])
            t = time.perf_counter()
            gf.CreateStructure(copy_back=False)
            best = min(best, time.perf_counter() - t)
        return best

    spread = cost("any")
    # sorted by the whole list: a few times the work of the row-wise form; a warp
    # that sorts the row by itself takes some three hundred times as long
    assert cost("one face") <= 20 * spread
    assert cost("one node") <= 20 * spread
    gf.close()
