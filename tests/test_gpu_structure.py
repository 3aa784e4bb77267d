"""The merge of contact lists into the pattern at the sizes where its per-row
sort and scan change form: no contact, one, rows with up to 32 codes, rows with
more, one row in every contact, lists that grow, shrink, repeat and end.  The
pattern, the slot maps and the assembled system against the oracle."""
import numpy as np
import pytest

from icflow_b200 import mesh as M
from icflow_b200.model_prms import config_prms
from tests.harness import Oracle, compare, gpu_assemble, oracle_assemble, orc_prms_from, random_state

pytestmark = pytest.mark.gpu


def _contacts(coll, kind, n, rng):
    """n (node, face) contacts: faces of the mesh, nodes off their face."""
    free = np.nonzero(coll.alt >= 0)[0]
    faces = coll.faces[rng.integers(0, len(coll.faces), n)]
    nodes = rng.integers(0, len(coll.x0), n)
    if kind == "one node":
        nodes[:] = free[len(free) // 2]
    elif kind == "one face":
        faces[:] = coll.faces[len(coll.faces) // 2]
    elif kind == "last row":
        nodes[:] = free[-1]
    elif kind == "repeated":
        nodes[n // 2:], faces[n // 2:] = nodes[:n - n // 2], faces[:n - n // 2]
    ok = ~(faces == nodes[:, None]).any(axis=1)
    return np.concatenate([nodes[:, None], faces], axis=1)[ok].astype(np.int32)


LISTS = [("any", 1), ("any", 7), ("one node", 8), ("one node", 9), ("one face", 33), ("any", 0), ("any", 900),
         ("one node", 700), ("one face", 1500), ("last row", 40), ("repeated", 64), ("any", 5000), ("any", 3)]


def test_contact_lists_of_every_size():
    coll = M.cantilever()
    O = Oracle()
    prms = config_prms(penaltyK=1e8)
    p = orc_prms_from(O, prms)
    from icflow_b200.gpu_functionality import GPU_Functionality

    gf = GPU_Functionality(0)
    gf.prms = prms
    gf.mc = coll
    gf.SetConstants()
    gf.TransferStaticDataToDevice()
    nc = len(coll.czs)
    state = random_state(coll, 0, du=2e-6)
    zero = np.zeros((nc, 3))
    rng = np.random.default_rng(5)
    for kind, n in LISTS:
        imp = _contacts(coll, kind, n, rng)
        g = gpu_assemble(gf, coll, state, 1e-4, zero, zero, np.zeros(nc, np.int32), impacts=imp)
        o = oracle_assemble(O, p, coll, state, 1e-4, zero, zero, imp)
        compare(g, o)
    gf.close()
