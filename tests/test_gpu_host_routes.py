"""
The host call on pageable arrays (qpd_run_host): which way the chunks go for the packing threads there are, and the same
volume, bit for bit, as the inputs packed on the device give, with chunks that the volume does not fill.

A chunk packed on the device shows as a launch of the pack kernel.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def plan_of(case):
    from qpop_diffraction_b200 import Plan, crystal_from
    p = case.params
    plan = Plan(case.shape, (p.dx, p.dy, p.dz), p.nPhase, p.nStruc)
    plan.set_crystal(crystal_from(p, case.atoms))
    return plan


# one whole chunk; one cell less; a last chunk of 95 cells, and of 6; four even ones
@pytest.mark.parametrize("shape", [(64, 64, 16), (257, 255, 1), (131, 501, 1), (331, 18, 33), (61, 67, 97)])
@pytest.mark.parametrize("weights", ["onehot", "region", "dense"])
@pytest.mark.parametrize("threads", [1, 2, 16])
def test_pageable_arrays(gpu, monkeypatch, shape, weights, threads):
    torch = gpu
    from qpop_diffraction_b200 import workloads
    monkeypatch.setenv("QPOP_B200_HOST_THREADS", str(threads))
    case = workloads.random_case(shape, seed=sum(shape), nPhase=2, weights=weights)
    t = lambda a: torch.from_numpy(a).to("cuda:0")
    with plan_of(case) as plan:
        want = plan.run_device(plan.pack(t(case.oPhase), t(case.oStruc), t(case.u), t(case.region))).cpu().numpy()
        plan.enable_timing(True)
        for _ in range(3):
            got = plan.run_host(case.oPhase, case.oStruc, case.u, case.region)
            np.testing.assert_array_equal(got, want)
        packed_on_device = "pack" in plan.stage_times()
        plan.device_status()
    # a thread that packs alone is slower than the driver's copies: its chunks may go the device way
    assert packed_on_device == (threads == 1)
