"""
The float32 and float64 passes at sizes where their tiles are the ones of real volumes: tiles of 8 and more pencils with
a partial last one, z stages whose CTAs walk several tiles, and every compiled length once, against the general kernels
(QPOP_B200_GENERIC=1); order-parameter components fewer than three; more fold inputs than one pass takes.

Tolerances as between any two float32 volumes that meet the contract of 1e-5 I_max each: 2e-5 of the largest value,
1e-9 in float64.
"""

import re
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CSRC = Path(__file__).resolve().parents[1] / "q-pop-diffraction_b200" / "csrc"
AXIS_LENGTHS = sorted(int(n) for n in re.findall(r"\bX\((\d+),", (CSRC / "qpd_axisct_lengths.h").read_text()))
Z_LENGTHS = sorted(int(a) * int(b) for a, b in re.findall(
    r"\bX\((\d+), (\d+)\)", (CSRC / "qpd_zcol.cu").read_text().split("#define QPD_ZCOL_LENGTHS(X)")[1].split("\n\n")[0]))
TOL = {"fp32": 2e-5, "fp64": 1e-9}


def plan_of(case, precision="fp32"):
    from qpop_diffraction_b200 import Plan, crystal_from
    p = case.params
    plan = Plan(case.shape, (p.dx, p.dy, p.dz), p.nPhase, p.nStruc, precision=precision)
    plan.set_crystal(crystal_from(p, case.atoms))
    return plan


def outputs(torch, case, precision="fp32", adjoint=True, cta_tiles=0):
    t = lambda a: torch.from_numpy(a).to("cuda:0")
    with plan_of(case, precision) as plan:
        plan.set_cta_tiles(cta_tiles)
        inputs = plan.pack(t(case.oPhase), t(case.oStruc), t(case.u), t(case.region))
        got = [plan.run_device(inputs).clone()]
        if adjoint:
            got += plan.adjoint(inputs, t(np.random.default_rng(5).normal(size=plan.n)))
        plan.device_status()
    return got


def assert_close(got, want, tol):
    for a, b in zip(got, want):
        assert (a.double() - b.double()).abs().max() <= tol * b.double().abs().max()


def against_general(torch, monkeypatch, case, precision="fp32", adjoint=True):
    monkeypatch.setenv("QPOP_B200_GENERIC", "0")
    got = outputs(torch, case, precision, adjoint)
    monkeypatch.setenv("QPOP_B200_GENERIC", "1")
    assert_close(got, outputs(torch, case, precision, adjoint), TOL[precision])


def test_the_lists_are_read():
    assert len(AXIS_LENGTHS) == len(set(AXIS_LENGTHS)) == 200 and len(Z_LENGTHS) == len(set(Z_LENGTHS)) == 47


# pencils per tile and what is left of the last one, in the y and x passes of the runtime-length kernels
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("shape,weights", [
    ((275, 34, 75), "region"),    # y: 32 pencils of 34 rows; x: 8 of 275, 6 left
    ((34, 605, 75), "onehot"),    # y: 8 of 605 (16 values per thread), 6 left
    ((605, 51, 49), "dense"),     # x: 8 of 605, 3 left
    ((1331, 3, 225), "region"),   # x: 4 of 1331, 3 left
    ((45, 34, 100), "dense"),     # z: 4 columns of 100, 2 left
    ((75, 68, 22), "onehot")])    # z: 16 columns of 22, 12 left
def test_runtime_length_tiles(gpu, monkeypatch, shape, weights, precision):
    from qpop_diffraction_b200 import workloads
    case = workloads.random_case(shape, seed=sum(shape), nPhase=2, weights=weights)
    against_general(gpu, monkeypatch, case, precision)


# several tiles per CTA, the number of columns (9009) no multiple of a tile's: odd nz, twiddled and coprime factors, pairs
@pytest.mark.parametrize("nz", [49, 60, 64, 75, 88, 105, 128, 136])
@pytest.mark.parametrize("weights,phases", [("region", 2), ("onehot", 3)])
def test_z_stage_walks_tiles(gpu, monkeypatch, nz, weights, phases):
    from qpop_diffraction_b200 import workloads
    case = workloads.random_case((99, 91, nz), seed=nz, nPhase=phases, weights=weights)
    k = np.random.default_rng(nz).uniform(-0.02, 0.05, size=(phases, case.atoms.nAtom))
    if weights == "region":
        case.atoms.su1, case.atoms.su2, case.atoms.su3 = workloads.isotropic_shifts(k)
    against_general(gpu, monkeypatch, case, adjoint=False)
    monkeypatch.setenv("QPOP_B200_GENERIC", "0")
    walk, one = (outputs(gpu, case, adjoint=False, cta_tiles=t)[0] for t in (0, 1))
    assert gpu.equal(walk, one)


@pytest.mark.parametrize("n", AXIS_LENGTHS)
def test_every_compiled_axis_length(gpu, monkeypatch, n):
    from qpop_diffraction_b200 import workloads
    for shape in ((n, 3, 10), (3, n, 9)):
        against_general(gpu, monkeypatch, workloads.random_case(shape, seed=n, nPhase=2, weights="region"))


@pytest.mark.parametrize("nz", Z_LENGTHS)
def test_every_compiled_z_length(gpu, monkeypatch, nz):
    from qpop_diffraction_b200 import workloads
    against_general(gpu, monkeypatch, workloads.random_case((11, 5, nz), seed=nz, nPhase=2, weights="region"), adjoint=False)


@pytest.mark.parametrize("nStruc", [0, 1, 2])
@pytest.mark.parametrize("shape", [(99, 91, 64), (24, 35, 75), (18, 20, 50)])
def test_fewer_components(gpu, monkeypatch, shape, nStruc):
    """P holds nStruc planes and no more."""
    from qpop_diffraction_b200 import workloads
    case = workloads.random_case(shape, seed=7, nPhase=2, weights="region")
    case.params.nStruc = nStruc
    for k in ("su1", "su2", "su3"):
        setattr(case.atoms, k, getattr(case.atoms, k)[:nStruc])
    t = lambda a: gpu.from_numpy(a).to("cuda:0")
    got = []
    for generic in ("0", "1"):
        monkeypatch.setenv("QPOP_B200_GENERIC", generic)
        with plan_of(case) as plan:
            n = plan.n
            inputs = plan.pack(t(case.oPhase), t(case.oStruc[:nStruc * n]), t(case.u), t(case.region))
            inputs["P"] = inputs["P"][:max(nStruc, 1) * n].clone()
            got.append([plan.run_device(inputs).clone(), *plan.adjoint(inputs, t(np.random.default_rng(5).normal(size=n)))])
            plan.device_status()
    for a, b in zip(*got):
        assert (a.double() - b.double()).abs().max() <= TOL["fp32"] * b.double().abs().max()


@pytest.mark.parametrize("atoms", [21, 22, 24])
def test_more_fold_inputs_than_a_pass_takes(gpu, monkeypatch, atoms):
    """21 atoms with an (R_x, R_y) each make 63 inputs of the y pass; 22 make 66, which the general kernels take."""
    from qpop_diffraction_b200 import workloads
    case = workloads.random_case((24, 34, 20), seed=atoms, nPhase=1, weights="onehot", nAtom=atoms)
    case.atoms.xAtom = np.random.default_rng(atoms).uniform(size=(atoms, 3))
    case.atoms.xAtom[:, 0] = np.arange(atoms) % 5 / 5 + 0.05  # five R_x, so that the fused schedule holds them
    for precision in ("fp32", "fp64"):
        against_general(gpu, monkeypatch, case, precision)


@pytest.mark.parametrize("shape,n", [((16384, 1, 1), 16384), ((1, 9000, 1), 9000), ((1, 1, 4096), 4096)])
def test_no_tables_for_lengths_beyond_the_tiles(gpu, shape, n):
    """An axis longer than any tile of the runtime-length passes holds its N twiddles and no rows for those passes."""
    from qpop_diffraction_b200 import Plan
    with Plan(shape, (0.4, 0.4, 0.4), 1) as plan:
        rest = 256 + 2 * 2 * 8  # the status word, and the tables of two axes of length 1
        assert plan.workspace_bytes == 8 * n + rest
