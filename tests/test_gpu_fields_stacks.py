"""
Field preparation on the GPU over stacks that its blocks share out differently: crops that start many layers up, planes
whose columns fill no whole block, blocks of one chunk of layers and of several, a last block with fewer.

Bit-exact with qpd_pack_device on the oracle-prepared float64 arrays, as in test_gpu_fields.py.
"""

import numpy as np
import pytest

from test_gpu_fields import pack_both

pytestmark = pytest.mark.gpu


# (nx, ny, nz), z0, layers of the stack: chunks x column blocks in the comment
@pytest.mark.parametrize("shape,z0,full", [
    ((33, 7, 40), 70, 118),         # 2 x 8, deep: a block per chunk that sums two chunks below
    ((5, 3, 33), 0, 33),            # 2 x 1
    ((45, 45, 1280), 37, 1330),     # 41 x 64: two chunks per block, the last block one
    ((239, 241, 70), 30, 100),      # 4 x 1800: one block walks all, the first and last in part
    ((241, 239, 60), 64, 124),      # 2 x 1800, deep: one block walks both
    ((239, 241, 61), 3, 64)])       # 2 x 1800 from layer 0: a block per chunk
@pytest.mark.parametrize("phase_file", [False, True])
def test_stacks(gpu, shape, z0, full, phase_file):
    from qpop_diffraction_b200 import Plan
    rng = np.random.default_rng(sum(shape))
    nx, ny, nz = shape
    f = lambda *s: rng.standard_normal(s, dtype=np.float32)
    mat = rng.integers(0, 3, size=(full, ny, nx)).astype(np.int8)
    region = rng.random((nz, ny, nx), dtype=np.float32)
    phase = None
    if phase_file:
        a = rng.random((nz, ny, nx), dtype=np.float32)
        phase = np.stack([a, 1 - a])
    case = dict(P=f(3, nz, ny, nx), u=f(3, nz, ny, nx) * np.float32(2e-11), phase=phase, region=region, mat=mat, z0=z0,
                dc=np.array([-0.0125, 0.0, 0.0213]), phase_of=np.array([0, -1, 1], dtype=np.int32), ramp_dz=0.41)
    with Plan(shape, (0.4, 0.4, 0.41), 2) as plan:
        got, want, _ = pack_both(gpu, plan, case)
        for key in ("P", "U", "phase", "weight", "wdense"):
            assert (got[key] is None) == (want[key] is None), key
            if got[key] is not None:
                assert gpu.equal(got[key], want[key]), key
        # a bad index in the first and in the last layer of the stack below the crop's end, in the last column
        for layer in (0, z0 + nz - 1):
            bad = mat.copy()
            bad[layer, ny - 1, nx - 1] = 3
            d = lambda a: gpu.from_numpy(np.ascontiguousarray(a)).to("cuda:0")
            with pytest.raises(ValueError):
                plan.pack_fields(d(case["P"]), d(bad), case["dc"], case["phase_of"], case["ramp_dz"], z0=z0)
