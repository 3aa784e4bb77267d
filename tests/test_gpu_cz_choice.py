"""Which cohesive-zone kernel runs, and under which name it is reported: every
variant is one kernel, and without one chosen the model's size decides."""
import numpy as np
import pytest

from icflow_b200 import mesh as M
from icflow_b200.model_prms import config_prms
from tests.harness import random_state

NAMES = {"k_cz_gp", "k_cz_lane"}


def test_both_kernels_have_the_zones_bytes():
    from bench import kernel_share_bytes

    for name in NAMES:
        assert kernel_share_bytes(name, 1, 1, 1, 1, 1000, 1) == 240000


@pytest.mark.gpu
@pytest.mark.parametrize("n, grains, automatic", [(6, 5, "k_cz_gp"), (32, 128, "k_cz_lane")])
def test_zone_kernel_by_size_and_by_variant(n, grains, automatic):
    from icflow_b200.gpu_functionality import GPU_Functionality

    coll = M.polycrystal(n=n, grains=grains, seed=0)
    gf = GPU_Functionality(0)
    gf.prms = config_prms(penaltyK=1e8)
    gf.mc = coll
    gf.SetConstants()
    gf.TransferStaticDataToDevice()
    nc = len(coll.czs)
    assert (nc > 23680) == (automatic == "k_cz_lane")
    gf.TransferNodesToGPU(*random_state(coll, 3, du=4e-6))
    gf.TransferPCSR(np.zeros((nc, 3)), np.zeros((nc, 3)), np.zeros(nc, np.int32))
    gf.CreateStructure()

    def ran():
        return {k["name"] for k in gf.ProfileAssembly(1e-4, reps=1)} & NAMES

    assert ran() == {automatic}
    for variant, name in enumerate(["k_cz_gp", "k_cz_gp", "k_cz_gp", "k_cz_lane"]):
        gf.SetVariant(4, variant)
        assert ran() == {name}, variant
    timed = [r["variant"] for r in gf.Autotune(1e-4, reps=2) if r["kernel"] == "k_cz_gp"]
    assert len(timed) == len(set(timed)) == 4
    gf.close()
