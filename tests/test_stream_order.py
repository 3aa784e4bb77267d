"""Uploads and fills are ordered with the work that uses them.  A context's work
runs on a stream of its own that does not wait for the null stream, and a copy
from pageable memory or a fill on the null stream may return before it has run:
neither may be used in the library, and work pending on the default stream of
the host program changes no result.  A network's stream is of the same kind."""
import re
from pathlib import Path

import numpy as np
import pytest

from icflow_b200 import mesh as M
from icflow_b200.model_prms import config_prms
from tests.harness import random_state

CSRC = Path(__file__).resolve().parents[1] / "icflow_b200" / "csrc"
SOURCES = sorted(p.name for p in [*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")])


@pytest.mark.parametrize("name", SOURCES)
def test_no_upload_or_fill_on_the_null_stream(name):
    text = re.sub(r"//[^\n]*", "", (CSRC / name).read_text())
    assert not re.findall(r"\bcudaMemset\s*\(", text)
    assert not [c for c in re.findall(r"\bcudaMemcpy\s*\([^;]*;", text) if "DeviceToHost" not in c]


def pending_work():
    """Some 100 ms of matrix products on the default stream, enqueued."""
    import torch

    a = torch.ones((4096, 4096), device="cuda")
    b = torch.empty_like(a)
    torch.mm(a, a, out=b)
    torch.cuda.synchronize()
    for _ in range(60):
        torch.mm(a, a, out=b)
    return a, b


def _values(coll, busy):
    from icflow_b200.gpu_functionality import GPU_Functionality

    rng = np.random.default_rng(2)
    nn, nc = len(coll.x0), len(coll.czs)
    u, v, a, du = (rng.random((nn, 3)) for _ in range(4))
    pmax = rng.random((nc, 3)) * 2e-6
    failed = (rng.random(nc) < 0.1).astype(np.int32)
    gf = GPU_Functionality(0)
    gf.prms = config_prms(penaltyK=1e8)
    gf.mc = coll
    gf.SetConstants()
    keep = pending_work() if busy else None
    gf.TransferStaticDataToDevice()
    gf.SetNodeState(u, v, a)
    gf.SetDU(du)
    gf.TransferPCSR(pmax, pmax[:, ::-1].copy(), failed)
    gf.TransferNodesToGPU(*random_state(coll, 3, du=4e-6))
    if busy:
        import torch

        torch.cuda.synchronize()
        del keep
    got = gf.GetNodeState()
    for x, y in zip(got, (u, v, a, du)):
        assert np.array_equal(x, y)
    gf.SetImpacts(np.zeros((0, 4), np.int32))
    gf.CreateStructure()
    gf.AssembleElemsAndCZs(1e-4)
    vals, rhs = (x.copy() for x in gf.TransferLinearSystemToHost())
    tent, flags, avg = gf.GetCZTentative()
    state = gf.TransferUpdatedStateToHost()
    gf.close()
    return dict(state, vals=vals, rhs=rhs, tent=tent, flags=flags, avg_tent=avg)


@pytest.mark.gpu
def test_static_data_under_pending_work():
    coll = M.polycrystal(n=6, grains=5, seed=4, platens=True, gap=-0.3)
    a, b = _values(coll, False), _values(coll, True)
    for k in a:
        assert np.array_equal(a[k], b[k]), k


def _network(busy):
    from icflow_b200.warm_start import MLP, NI, NO, init_params

    rng = np.random.default_rng(4)
    p, norm = init_params(1), np.concatenate([rng.normal(size=NI), rng.uniform(0.5, 2, NI), np.ones(NO)])
    x = rng.normal(size=(5000, NI)).astype(np.float32)
    t = rng.normal(size=(5000, NO)).astype(np.float32)
    keep = pending_work() if busy else None
    net = MLP()
    net.set_params(p, norm.astype(np.float32))
    g0, l0 = net.grad(x, t)
    loss = net.train(x, t, epochs=2, batch=512, lr=1e-3, seed=3)
    q = net.get_params()[0]
    net.set_params(p, norm.astype(np.float32))  # and the moments start from zero again
    again = net.train(x, t, epochs=2, batch=512, lr=1e-3, seed=3)
    net.close()
    del keep
    assert loss == again
    return g0, l0, loss, q


@pytest.mark.gpu
def test_network_under_pending_work():
    for a, b in zip(_network(False), _network(True)):
        assert np.array_equal(a, b)
