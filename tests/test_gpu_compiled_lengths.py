"""
The compile-time z stage (csrc/qpd_zcol.cuh) and y and x passes (csrc/qpd_axisct.cuh) of the float32 path, at the
edges of their tiles: column counts that a tile does not divide, z extents that leave a partial chunk or are odd, isotropic and
general ionic shifts, one to three phases, cells that do not scatter, fractional weights.

Tolerances: the float32 contract against the oracle (max |dI| / I_max <= 1e-5, relative error <= 1e-3 above
1e-6 I_max); between these kernels and the general ones both errors add: 2e-5 of the largest value.
"""

import numpy as np
import pytest

from conftest import fp32_errors

pytestmark = pytest.mark.gpu


def make_case(shape, phases, weights, iso, seed):
    from qpop_diffraction_b200 import workloads
    case = workloads.random_case(shape, seed=seed, nPhase=phases, weights=weights, strain=True)
    if iso:
        k = np.random.default_rng(seed).uniform(-0.02, 0.05, size=(phases, case.atoms.nAtom))
        case.atoms.su1, case.atoms.su2, case.atoms.su3 = workloads.isotropic_shifts(k)
    return case


def plan_of(case):
    from qpop_diffraction_b200 import Plan, crystal_from
    p = case.params
    plan = Plan(case.shape, (p.dx, p.dy, p.dz), p.nPhase, p.nStruc)
    plan.set_crystal(crystal_from(p, case.atoms))
    return plan


@pytest.mark.parametrize("iso", [True, False])
@pytest.mark.parametrize("nz", [16, 20, 25, 30, 32, 42, 45, 49, 56, 60, 64, 68, 72, 75, 85, 88, 90, 96, 102, 104, 105, 119, 120, 128, 136])
def test_z_stage(gpu, nz, iso):
    from oracle import diffraction_oracle as oracle
    for shape, phases, weights in (((1, 1, nz), 1, "onehot"), ((3, 5, nz), 2, "region"), ((7, 9, nz), 3, "onehot")):
        case = make_case(shape, phases, weights, iso, seed=sum(shape))
        ref = oracle.diffraction(*case.args())[0]
        with plan_of(case) as plan:
            plan.set_cta_tiles(2 if phases == 3 else 0)
            I = plan.run_host(case.oPhase, case.oStruc, case.u, case.region)
            plan.device_status()
        dmax, rel = fp32_errors(I, ref)
        assert dmax <= 1e-5 and rel <= 1e-3, (shape, dmax, rel)


@pytest.mark.parametrize("N", [24, 35, 48, 63, 64, 68, 100, 117, 120, 128, 135, 150, 195, 200, 225, 240, 256, 289, 300, 390, 400, 512,
                               600, 768, 900, 1024])
def test_axis_passes(gpu, monkeypatch, N):
    """Both strided positions, whole and partial z chunks; the volume against the oracle, the gradient against the
    general kernels (QPOP_B200_GENERIC=1)."""
    torch = gpu
    from oracle import diffraction_oracle as oracle
    dev = torch.device("cuda", 0)
    t = lambda x: torch.from_numpy(x).to(dev)
    for shape in ((N, 3, 2), (2, N, 10), (N, 2, 9), (3, N, 7)):
        case = make_case(shape, 2, "region", False, seed=sum(shape))
        ref = oracle.diffraction(*case.args())[0]
        g = torch.from_numpy(np.random.default_rng(2).normal(size=shape)).to(dev)
        got = []
        for generic in ("0", "1"):
            monkeypatch.setenv("QPOP_B200_GENERIC", generic)
            with plan_of(case) as plan:
                inputs = plan.pack(t(case.oPhase), t(case.oStruc), t(case.u), t(case.region))
                I = plan.run_device(inputs).clone()
                dP, dU = plan.adjoint(inputs, g)
                got.append([x.double().cpu().numpy() for x in (I, dP, dU)])
                plan.device_status()
        dmax, rel = fp32_errors(got[0][0], ref)
        assert dmax <= 1e-5 and rel <= 1e-3, (shape, dmax, rel)
        for a, b in zip(got[0][1:], got[1][1:]):
            assert np.abs(a - b).max() <= 2e-5 * np.abs(b).max()
