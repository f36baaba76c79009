"""
The work a user of this package has it do, as cases that can be timed one by one.

Every case goes through the public entry points (``Plan``, ``autograd.intensity``,
``diffraction``, ``serving.Engine``) on seeded synthetic films: a polar-vortex or stripe texture
with noise, a strain gradient growing up z and smooth displacement, the 5-atom perovskite cell.
A program that computes in float32 also keeps its volumes in float32, so those passes end with
the conversion of I (whose float64 values carry float32 amplitudes); float64 plans return I as it is.
"""

import math
from types import SimpleNamespace

import numpy as np
import torch

DEV = "cuda"
CELL = (0.39, 0.39, 0.40)  # nm, the perovskite cell and the grid spacing
ATOMS = np.array([[0.0, 0.0, 0.0], [0.5, 0.5, 0.5], [0.5, 0.5, 0.0], [0.5, 0.0, 0.5], [0.0, 0.5, 0.5]])
HKLS = ((0, 0, 2), (1, 0, 3), (1, 1, 3), (2, 0, 0))


def listed():
    return [
        # one small volume: a quick look at a test cell, where launches and latency count
        dict(name="volume_64x64x32", kind="volume", nx=64, ny=64, nz=32, phases=1, weights="onehot", precision="fp32"),
        # a 2-D phase-field film, straight from the simulation's own float32 fields in file order
        dict(name="film_1x400x400", kind="film", nx=1, ny=400, nz=400, phases=1, weights="onehot", precision="fp32"),
        # the drop-in call on float64 host arrays, as the command-line program makes it
        dict(name="host_96x96x64", kind="host", nx=96, ny=96, nz=64, phases=2, weights="onehot", precision="fp32"),
        # an odd-sized crop with a fractional region weight
        dict(name="volume_150x135x75", kind="volume", nx=150, ny=135, nz=75, phases=2, weights="region", precision="fp32"),
        # overlapping phase fractions of a diffuse interface
        dict(name="volume_240x200x60_dense", kind="volume", nx=240, ny=200, nz=60, phases=2, weights="dense", precision="fp32"),
        # a converged float64 volume, to check a float32 one against
        dict(name="volume_128x128x64_fp64", kind="volume", nx=128, ny=128, nz=64, phases=2, weights="onehot", precision="fp64"),
        # one snapshot seen at four reflections, the tables set for each
        dict(name="scan_128x128x128", kind="scan", nx=128, ny=128, nz=128, phases=2, weights="onehot", precision="fp32"),
        # requests of two grids in flight together
        dict(name="serving_mix", kind="serving", nx=256, ny=256, nz=64, phases=2, weights="onehot", precision="fp32"),
        # one step of fitting fields to a measured map: intensity and its gradient
        dict(name="gradient_256x256x64", kind="gradient", nx=256, ny=256, nz=64, phases=2, weights="onehot", precision="fp32"),
        dict(name="gradient_120x100x50", kind="gradient", nx=120, ny=100, nz=50, phases=2, weights="region", precision="fp32"),
        # the two-phase film, and the largest grid that is served
        dict(name="volume_512x512x104", kind="volume", nx=512, ny=512, nz=104, phases=2, weights="onehot", precision="fp32"),
        dict(name="volume_1024x1024x68", kind="volume", nx=1024, ny=1024, nz=68, phases=2, weights="onehot", precision="fp32"),
    ]


# Grids that the configurations and tests of this repository name; a draw takes one of these lengths or any other.
ROUND_XY = (32, 64, 128, 256, 512, 1024)
ROUND_Z = (32, 64, 68, 104, 128)


def _smooth(n):
    """Whether n is a product of primes up to 17, as the grids of a spectral phase-field solver are."""
    for p in (2, 3, 5, 7, 11, 13, 17):
        while n % p == 0:
            n //= p
    return n == 1


def _length(rng, lo, hi, round_ones):
    if rng.random() < 0.35:
        some = [n for n in round_ones if lo <= n <= hi]
        if some:
            return rng.choice(some)
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    while not _smooth(n) and n < hi:  # the next grid a solver would run on; odd ones among them
        n += 1
    return n if _smooth(n) else hi


def draw(rng):
    kind = rng.choice(("volume", "volume", "volume", "gradient", "gradient", "scan", "film", "host", "serving"))
    precision = "fp64" if kind == "volume" and rng.random() < 0.2 else "fp32"
    weights = rng.choice(("onehot", "onehot", "region", "dense")) if kind in ("volume", "gradient", "host") else "onehot"
    most = {"volume": 30e6, "gradient": 6e6, "scan": 4e6, "film": 2e6, "host": 1e6, "serving": 4e6}[kind]
    most = min(most, 2.5e6) if precision == "fp64" or weights == "dense" else most
    while True:
        nx, ny = (_length(rng, 24, 1024, ROUND_XY) for _ in range(2))
        nz = _length(rng, 16, 160, ROUND_Z)
        if kind == "film" and rng.random() < 0.5:
            nx, ny, nz = 1, _length(rng, 100, 1024, ROUND_XY), _length(rng, 40, 512, ROUND_Z)
        if 20_000 <= nx * ny * nz <= most:
            break
    return dict(kind=kind, nx=nx, ny=ny, nz=nz, phases=rng.choice((1, 2)) if weights != "dense" else 2,
                weights=weights, precision=precision)


# ---- inputs, from the seed alone


def _shape(case):
    return case["nx"], case["ny"], case["nz"]


def _params(case, shape=None):
    nx, ny, nz = shape or _shape(case)
    return SimpleNamespace(nx=nx, ny=ny, nz=nz, n=nx * ny * nz, dx=CELL[0], dy=CELL[1], dz=CELL[2],
                           nPhase=case["phases"], nStruc=3, strainAvg=np.zeros(6))


def _atoms(case, seed, hkl):
    """Perovskite cell: Cromer-Mann-like form factors and ionic shifts along P, per phase and atom."""
    rng = np.random.default_rng([seed] + list(hkl))
    aC, NP, NA = np.diag(CELL), case["phases"], len(ATOMS)
    f = rng.uniform(5.0, 60.0, (NP, NA)) + 1j * rng.uniform(0.0, 2.0, (NP, NA))
    k = rng.uniform(-0.02, 0.05, (NP, NA))
    su = [np.zeros((3, NP, NA)) for _ in range(3)]
    for d in range(3):
        su[d][d] = k
    q00 = np.asarray(hkl, dtype=np.float64) @ (2 * math.pi * np.linalg.inv(aC).T)
    return SimpleNamespace(aC=aC, q00=q00, xAtom=ATOMS, nAtom=NA, fAtom=f, su1=su[0], su2=su[1], su3=su[2])


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _texture(shape, seed):
    """P and u of a film, (3, nx, ny, nz) float32 each."""
    nx, ny, nz = shape
    g, f32 = _gen(seed), dict(dtype=torch.float32, device=DEV)
    x, y, z = torch.arange(nx, **f32).view(-1, 1, 1), torch.arange(ny, **f32).view(1, -1, 1), torch.arange(nz, **f32)
    P = torch.empty((3, nx, ny, nz), **f32).normal_(0.0, 0.02, generator=g)
    film = (z >= nz // 4).to(torch.float32)
    if seed % 2:  # a1/a2 stripes
        a1 = (((x + y) % 16) < 8).to(torch.float32)
        P[0] += 0.5 * a1 * film
        P[1] += 0.5 * (1 - a1) * film
    else:  # vortices rotating in x (or y, in a film of one x layer) and z
        k = 2 * math.pi / 10
        s = x if nx > 1 else y
        a, b = torch.sin(k * s) * torch.cos(k * z), torch.cos(k * s) * torch.sin(k * z)
        r = torch.clamp(torch.sqrt(a * a + b * b), min=1e-12)
        P[0] += 0.6 * a / r * film
        P[2] -= 0.6 * b / r * film
    m = torch.rand(12, generator=g, **f32)
    wave = [2 * math.pi * (x * round(4 * float(m[3 * d])) / nx + y * round(4 * float(m[3 * d + 1])) / ny +
                           z * round(4 * float(m[3 * d + 2])) / nz) for d in range(3)]
    u = torch.empty((3, nx, ny, nz), **f32).normal_(0.0, 0.0005, generator=g)
    for d in range(3):
        u[d] += 0.005 * torch.cos(wave[d] + 6.0 * m[9 + d])
    e = 0.01 * z / max(nz - 1, 1)
    u[2] += (torch.cumsum(e, 0) - 0.5 * e) * CELL[2]
    return P, u


def _weights(case, shape, seed):
    """Phase fractions (phases, nx, ny, nz) and region (nx, ny, nz), float32 values."""
    nx, ny, nz = shape
    g, f32, NP = _gen(seed + 7), dict(dtype=torch.float32, device=DEV), case["phases"]
    z = torch.arange(nz, **f32)
    sub = (z < nz // 4).to(torch.float32).expand(nx, ny, nz)
    region = torch.ones((nx, ny, nz), **f32)
    if case["weights"] == "dense":
        f = 0.5 + 0.5 * torch.tanh((z - nz / 4) / 4).expand(nx, ny, nz)
        f = f + 0.02 * torch.rand((nx, ny, nz), generator=g, **f32)
        oPhase = torch.stack([1.0 - 0.9 * f, 0.9 * f])
    elif NP == 1:
        oPhase = torch.ones((1, nx, ny, nz), **f32)
    else:
        oPhase = torch.stack([sub, 1 - sub])
    if case["weights"] != "onehot":
        region = 0.2 + 0.8 * torch.rand((nx, ny, nz), generator=g, **f32)
        region *= (torch.rand((nx, ny, nz), generator=g, **f32) > 0.1).to(torch.float32)
    return oPhase, region


def _fields(case, seed, shape=None):
    """oPhase, oStruc, u, region as flat float64 GPU tensors in the layout that diffraction() takes."""
    shape = shape or _shape(case)
    P, u = _texture(shape, seed)
    oPhase, region = _weights(case, shape, seed)
    return [t.double().reshape(-1) for t in (oPhase, P, u, region)]


def _film(case, seed):
    """Simulation fields in file order (nz, ny, nx), x fastest, and the material tables."""
    nx, ny, nz = _shape(case)
    P, u = _texture((nx, ny, nz), seed)
    back = lambda t: t.permute(2, 1, 0).contiguous()  # noqa: E731
    material = torch.ones((nz, ny, nx), dtype=torch.int8, device=DEV)
    material[: nz // 4] = 0
    phase_of = np.array([0, 1] if case["phases"] == 2 else [-1, 0], dtype=np.int32)
    return SimpleNamespace(P=[back(P[d]) for d in range(3)], u=[back(1e-9 * u[d]) for d in range(3)], material=material,
                           dc=np.array([0.0, 0.004 + 0.0001 * (seed % 5)]), phase_of=phase_of, dz=CELL[2])


def _loss_gradient(case, seed):
    """dL/dI of a weighted difference over the diffuse part of the map: the Bragg peak is masked out."""
    nx, ny, nz = _shape(case)
    f64 = dict(dtype=torch.float64, device=DEV)
    r2 = sum(((torch.arange(n, **f64) - n // 2) / 2.0).square().view([-1 if a == d else 1 for a in range(3)])
             for d, n in enumerate((nx, ny, nz)))
    w = torch.empty((nx, ny, nz), **f64).normal_(0.0, 1.0, generator=_gen(seed + 13))
    return w * (1 - torch.exp(-0.5 * r2))


SERVED = ((128, 128, 128), (256, 256, 64))


def _served_grids(case):
    return (SERVED[0], _shape(case)) if _shape(case) != SERVED[0] else (SERVED[1], _shape(case))


def prepare(case, seed):
    from qpop_diffraction_b200 import Plan, crystal_from
    s = SimpleNamespace(kind=case["kind"], fp64=case["precision"] == "fp64")
    params = _params(case)
    if s.kind == "host":
        s.params, s.atoms = params, _atoms(case, seed, HKLS[0])
        s.arrays = [t.cpu().numpy() for t in _fields(case, seed)]
        return s
    if s.kind == "serving":
        from qpop_diffraction_b200.serving import Engine, Request, Snapshot, SnapshotStore
        store = SnapshotStore()
        for i in range(4):
            shape = _served_grids(case)[i % 2]
            p = _params(case, shape)
            with Plan(shape, CELL, case["phases"]) as plan:
                store.add(Snapshot(i, "film", shape, p, plan.pack(*_fields(case, seed + i, shape))))
        s.engine = Engine(store, 16 << 30, crystal_of=lambda p, hkl: crystal_from(p, _atoms(case, seed, hkl)),
                          priorities=True, max_slots=2)
        s.requests = lambda: [Request(i, i % 4, HKLS[i // 4 + i % 2]) for i in range(8)]
        s.engine.run(s.requests() + s.requests())  # slots and graphs exist before the first request is served
        return s
    s.plan = Plan(_shape(case), CELL, case["phases"], precision=case["precision"])
    s.crystals = [crystal_from(params, _atoms(case, seed, hkl)) for hkl in HKLS]
    s.plan.set_crystal(s.crystals[0])
    if s.kind == "film":
        s.film = _film(case, seed)
        s.out = torch.empty(_shape(case), dtype=torch.float64, device=DEV)
        return s
    s.inputs = s.plan.pack(*_fields(case, seed))
    if s.kind == "gradient":
        s.P, s.U = (s.inputs[k].view((3,) + _shape(case)).requires_grad_(True) for k in ("P", "U"))
        s.g = _loss_gradient(case, seed)
    elif s.kind == "volume":
        s.out = torch.empty(_shape(case), dtype=torch.float64, device=DEV)
    return s


def run(s):
    if s.kind == "volume":
        I = s.plan.run_device(s.inputs, s.out)
        return I if s.fp64 else I.float()
    if s.kind == "film":
        f = s.film
        inputs = s.plan.pack_fields(f.P, f.material, f.dc, f.phase_of, f.dz, u=f.u)
        return s.plan.run_device(inputs, s.out).float()
    if s.kind == "scan":
        got = []
        for c in s.crystals:
            # the plan's tables are the ones the last volume reads: it has to be done before they are set again
            torch.cuda.current_stream().synchronize()
            s.plan.set_crystal(c)
            got.append(s.plan.run_device(s.inputs).float())
        return got
    if s.kind == "gradient":
        from qpop_diffraction_b200.autograd import intensity
        i = s.inputs
        I = intensity(s.plan, s.P, s.U, phase=i["phase"], weight=i["weight"], wdense=i["wdense"])
        dP, dU = torch.autograd.grad(I, (s.P, s.U), s.g)
        return I.float(), dP, dU
    if s.kind == "serving":
        got = {}

        def keep(request, I):  # on the slot's own stream, before its next request
            with torch.cuda.stream(request.slot.stream):
                got[str(request.id)] = I.float()

        for r in s.engine.run(s.requests(), result_of=keep):
            torch.cuda.current_stream().wait_stream(r.slot.stream)
        return got
    from qpop_diffraction_b200 import diffraction
    I, qx, qy, qz = diffraction(s.params, s.atoms, *s.arrays)
    return I.astype(np.float32), qx, qy, qz


def _cost(shape, case):
    """(bytes, operations) of one volume: inputs once, I once; source, transforms and fold of the grouped schedule."""
    n = shape[0] * shape[1] * shape[2]
    real = 8 if case["precision"] == "fp64" else 4
    w = {"onehot": 1, "region": 1 + real, "dense": case["phases"] * real}[case["weights"]]
    lg = [math.log2(max(m, 1)) for m in shape]
    ops = n * (5 * 60 + 5 * (20 * lg[2] + 12 * lg[1] + 4 * lg[0]) + 8 * 36 + 12)
    return n * (6 * real + w + 8 + (0 if real == 8 else 4)), ops


def work(case):
    n = case["nx"] * case["ny"] * case["nz"]
    b, f = _cost(_shape(case), case)
    kind = case["kind"]
    if kind == "scan":
        b, f = 4 * b, 4 * f
    elif kind == "film":
        b += n * 25
    elif kind == "gradient":  # the forward, its recomputation, and the transposed passes
        b, f = b + n * (8 + 24 + 24), 3 * f
    elif kind == "host":
        b = n * (8 * (case["phases"] + 7) + 8)
    elif kind == "serving":
        each = [_cost(s, case) for s in _served_grids(case)]
        b, f = 4 * sum(e[0] for e in each), 4 * sum(e[1] for e in each)
    return {"bytes": b, "flops": f}


# ---- what the model gives in 64 bits, in plain torch


def _model(shape, atoms, NP, oPhase, P, u, region):
    """I (nx, ny, nz) float64, fftshifted (oPhase, P, u, region as _fields gives them)."""
    n = shape[0] * shape[1] * shape[2]
    aC = atoms.aC
    B = 2 * math.pi * np.linalg.inv(aC).T
    G = np.round(aC @ atoms.q00 / (2 * math.pi)) @ B
    R, V = atoms.xAtom @ aC, float(np.linalg.det(aC))
    su = np.stack([atoms.su1, atoms.su2, atoms.su3])
    P, u, W = P.reshape(3, n), u.reshape(3, n), oPhase.reshape(NP, n) * region
    k = [torch.from_numpy(2 * math.pi * np.fft.fftfreq(m, h)).to(DEV).view([-1 if a == d else 1 for a in range(3)])
         for d, (m, h) in enumerate(zip(shape, CELL))]
    amp = 0
    for a in range(R.shape[0]):
        F = [0, 0, 0, 0]
        for p in range(NP):
            ua = [u[d] + sum(float(su[d, s, p, a]) * P[s] for s in range(3) if su[d, s, p, a]) for d in range(3)]
            e = W[p] * complex(atoms.fAtom[p, a]) * torch.exp(-1j * sum(float(G[d]) * ua[d] for d in range(3)))
            F = [F[0] + e] + [F[d + 1] + e * ua[d] for d in range(3)]
        shift = 1.0 / V
        for d in range(3):
            shift = shift * torch.exp(-1j * (k[d] + float(G[d])) * float(R[a, d]))
        F = [torch.fft.fftn(f.view(shape)) / n for f in F]
        amp = amp + shift * (F[0] - 1j * (k[0] * F[1] + k[1] * F[2] + k[2] * F[3]))
    S = 1.0
    for d, h in enumerate(CELL):
        S = S * torch.sinc(k[d] * h / (2 * math.pi))
    return torch.fft.fftshift(torch.clamp((S * amp).abs().square(), min=1e-50))


def exact(case, seed):
    shape, NP, kind = _shape(case), case["phases"], case["kind"]
    if kind == "film":
        f = _film(case, seed)
        there = lambda t: t.permute(2, 1, 0).double()  # noqa: E731
        dc = torch.from_numpy(f.dc).to(DEV)[there(f.material).long()]
        P = torch.stack([there(t) for t in f.P])
        u = torch.stack([there(t) * 1e9 for t in f.u])
        u[2] += (torch.cumsum(dc, 2) - 0.5 * dc) * f.dz
        ph = torch.from_numpy(f.phase_of).to(DEV)[there(f.material).long()]
        oPhase = torch.stack([(ph == p).double() for p in range(NP)])
        return _model(shape, _atoms(case, seed, HKLS[0]), NP, oPhase, P, u, 1.0)
    if kind == "serving":
        sets = [(g, _fields(case, seed + i, g)) for i, g in enumerate(_served_grids(case) * 2)]
        return {str(i): _model(sets[i % 4][0], _atoms(case, seed, HKLS[i // 4 + i % 2]), NP, *sets[i % 4][1]) for i in range(8)}
    oPhase, P, u, region = _fields(case, seed)
    if kind == "scan":
        return [_model(shape, _atoms(case, seed, hkl), NP, oPhase, P, u, region) for hkl in HKLS]
    atoms = _atoms(case, seed, HKLS[0])
    if kind == "gradient":
        P, u = P.requires_grad_(True), u.requires_grad_(True)
        I = _model(shape, atoms, NP, oPhase, P, u, region)
        dP, dU = torch.autograd.grad(I, (P, u), _loss_gradient(case, seed))
        return I.detach(), dP.view((3,) + shape), dU.view((3,) + shape)
    I = _model(shape, atoms, NP, oPhase, P, u, region)
    if kind == "host":
        return (I,) + tuple(np.fft.fftshift(2 * math.pi * np.fft.fftfreq(m, h)) + q
                            for m, h, q in zip(shape, CELL, atoms.q00))
    return I
