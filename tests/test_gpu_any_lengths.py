"""
The runtime-length passes (csrc/qpd_any.cuh) against the oracle, at the lengths where they can go wrong: every
radix from 2 to 17 on every axis, lengths of one to four stages, tiles that the pencils do not fill, fewer
pencils than a tile holds, z extents at the tile limits, and lengths that they leave to the general kernels.

Tolerances: the float32 contract (max |dI| / I_max <= 1e-5, relative error <= 1e-3 above 1e-6 I_max) and, for
float64, the reference's own rtol 1e-9 with atol 1e-12 I_max.  Between the passes and the general kernels both
errors add, so two float32 volumes differ by at most 2e-5 I_max.
"""

import numpy as np
import pytest

from conftest import fp32_errors

pytestmark = pytest.mark.gpu


def plan_of(case, precision):
    from qpop_diffraction_b200 import Plan, crystal_from
    p = case.params
    plan = Plan(case.shape, (p.dx, p.dy, p.dz), p.nPhase, p.nStruc, precision=precision)
    plan.set_crystal(crystal_from(p, case.atoms))
    return plan


def volume(case, precision):
    with plan_of(case, precision) as plan:
        I = plan.run_host(case.oPhase, case.oStruc, case.u, case.region)
        plan.device_status()
    return I


@pytest.mark.parametrize("shape", [
    (2, 3, 5), (6, 7, 9), (10, 11, 12), (13, 14, 15), (16, 17, 18), (19, 4, 8), (8, 23, 6),   # radices; 19, 23: general
    (1, 221, 3), (289, 1, 2), (3, 2, 225), (2, 3, 1023), (2, 2, 1025), (2, 2, 2040),          # 2 and 3 stages, z limits
    (5, 9, 33), (7, 33, 35), (45, 50, 49), (30, 300, 1), (343, 3, 7), (3, 1331, 2), (2, 2187, 1)])
def test_any_lengths(gpu, shape):
    from qpop_diffraction_b200 import workloads
    from oracle import diffraction_oracle as oracle
    for weights, phases in (("region", 2), ("dense", 2)):
        case = workloads.random_case(shape, seed=sum(shape), nPhase=phases, weights=weights, strain=True)
        ref = oracle.diffraction(*case.args())[0]
        np.testing.assert_allclose(volume(case, "fp64"), ref, rtol=1e-9, atol=1e-12 * ref.max())
        dmax, rel = fp32_errors(volume(case, "fp32"), ref)
        assert dmax <= 1e-5 and rel <= 1e-3, (dmax, rel)


@pytest.mark.parametrize("weights,phases,atoms", [("onehot", 1, None), ("region", 3, 7), ("dense", 3, 2)])
@pytest.mark.parametrize("shape", [(20, 18, 25), (9, 60, 14), (34, 5, 100)])
def test_any_equals_general(gpu, monkeypatch, shape, weights, phases, atoms):
    """The same volume and gradient as the general kernels (QPOP_B200_GENERIC=1), in every form of the inputs."""
    torch = gpu
    from qpop_diffraction_b200 import workloads
    case = workloads.random_case(shape, seed=sum(shape) + phases, nPhase=phases, weights=weights, nAtom=atoms)
    dev = torch.device("cuda", 0)
    t = lambda x: torch.from_numpy(x).to(dev)
    g = torch.from_numpy(np.random.default_rng(1).normal(size=shape)).to(dev)
    got = []
    for generic in ("0", "1"):
        monkeypatch.setenv("QPOP_B200_GENERIC", generic)
        for precision in ("fp32", "fp64"):
            with plan_of(case, precision) as plan:
                inputs = plan.pack(t(case.oPhase), t(case.oStruc), t(case.u), t(case.region))
                I = plan.run_device(inputs).clone()
                dP, dU = plan.adjoint(inputs, g)
                got.append([x.double().cpu().numpy() for x in (I, dP, dU)])
                plan.device_status()
    for k in range(3):
        for a, b, tol in ((got[0], got[2], 2e-5), (got[1], got[3], 1e-9)):
            assert np.abs(a[k] - b[k]).max() <= tol * np.abs(b[k]).max()
