"""
Two host threads, each with a plan of its own whose launches share kernels and differ in shared memory: every call
succeeds and gives the volume (and the gradient) that it gives alone, bit for bit.

The threads loop in a few lines of C, outside the interpreter's lock, so that their launches really meet.
"""

import ctypes
import shutil
import subprocess
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LOOP = r"""
typedef int (*call8)(void*, void*, void*, void*, void*, void*, void*, void*);
typedef int (*call10)(void*, void*, void*, void*, void*, void*, void*, void*, void*, void*);
extern "C" int loop(void* fn, void** a, int nargs, int n) {
    for (int i = 0; i < n; i++) {
        const int rc = nargs == 8 ? ((call8)fn)(a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7])
                                  : ((call10)fn)(a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7], a[8], a[9]);
        if (rc != 0) return rc;
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def loop(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ is needed to compile the loop")
    where = tmp_path_factory.mktemp("threads")
    (where / "loop.cpp").write_text(LOOP)
    subprocess.run([cxx, "-O2", "-shared", "-fPIC", str(where / "loop.cpp"), "-o", str(where / "loop.so")], check=True)
    return ctypes.CDLL(str(where / "loop.so")).loop


class Job:
    """One plan and its inputs; call(n) queues n volumes (or gradients) on a stream of its own."""

    def __init__(self, torch, loop, shape, weights, phases, precision="fp32", adjoint=False):
        from qpop_diffraction_b200 import Plan, crystal_from, workloads
        case = workloads.random_case(shape, seed=sum(shape), nPhase=phases, weights=weights)
        p = case.params
        self.plan = Plan(shape, (p.dx, p.dy, p.dz), phases, p.nStruc, precision=precision)
        self.plan.set_crystal(crystal_from(p, case.atoms))
        t = lambda a: torch.from_numpy(a).to("cuda:0")
        x = self.plan.pack(t(case.oPhase), t(case.oStruc), t(case.u), t(case.region))
        self.keep, self.loop, self.stream = x, loop, torch.cuda.Stream()
        n, dt = self.plan.n, self.plan.torch_dtype
        if adjoint:
            self.g = t(np.random.default_rng(3).normal(size=n))
            self.out = [torch.empty(3 * n, dtype=dt, device="cuda:0") for _ in range(2)]
            fn, last = self.plan.lib.qpd_adjoint_device, [self.g, *self.out]
        else:
            self.out = [torch.empty(n, dtype=torch.float64, device="cuda:0")]
            fn, last = self.plan.lib.qpd_run_device, self.out
        ptr = [v.data_ptr() if v is not None else None for v in (*(x[k] for k in ("P", "U", "phase", "weight", "wdense")), *last)]
        args = [self.plan._ctx.value, *ptr, self.stream.cuda_stream]
        self.args, self.fn = (ctypes.c_void_p * len(args))(*args), ctypes.cast(fn, ctypes.c_void_p)
        torch.cuda.synchronize()

    def call(self, n):
        rc = self.loop(self.fn, self.args, len(self.args), n)
        self.stream.synchronize()
        assert rc == 0, (self.plan.lib.qpd_last_error(self.plan._ctx) or b"").decode()
        return [o.clone() for o in self.out]


# one z stage with and without a weight array, and with few and many phases; the runtime-length passes at two lengths of
# one kernel; z stages of two lengths with dense weights; the adjoint; float64 z stages with few and many phases
@pytest.mark.parametrize("a,b", [
    (dict(shape=(8, 8, 104), weights="region", phases=2), dict(shape=(8, 8, 104), weights="onehot", phases=2)),
    (dict(shape=(8, 8, 60), weights="onehot", phases=6), dict(shape=(8, 8, 60), weights="onehot", phases=1)),
    (dict(shape=(1331, 3, 2), weights="region", phases=2), dict(shape=(1573, 3, 2), weights="region", phases=2)),
    (dict(shape=(3, 4, 1000), weights="dense", phases=2), dict(shape=(4, 3, 700), weights="dense", phases=2)),
    (dict(shape=(3, 2, 700), weights="region", phases=1, adjoint=True),
     dict(shape=(3, 3, 1001), weights="region", phases=1, adjoint=True)),
    (dict(shape=(8, 8, 64), weights="onehot", phases=6, precision="fp64"),
     dict(shape=(8, 8, 64), weights="onehot", phases=1, precision="fp64"))])
def test_two_plans_on_two_threads(gpu, loop, a, b):
    jobs = [Job(gpu, loop, **x) for x in (a, b)]
    alone = [j.call(1) for j in jobs]
    errors, barrier = [], threading.Barrier(2)

    def many(j, want):
        try:
            barrier.wait(30)
            assert all(gpu.equal(x, y) for x, y in zip(j.call(20000), want))
        except Exception as e:  # reported by the test's own thread
            errors.append(e)

    threads = [threading.Thread(target=many, args=x) for x in zip(jobs, alone)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for j in jobs:
        j.plan.close()
    assert not errors, errors
