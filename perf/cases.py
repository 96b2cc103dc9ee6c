"""Performance cases: the work a program has this package do, through its public entry points.

Each kind of case is one way the package is used:

* ``rollout``  one solver context: particles and coefficients set, a number of steps, results read
  back.  ``steps`` = 1 without a reset is the interactive frame loop.
* ``batch``    many instances of one or more domains stepped together, results read every few steps.
* ``serve``    a burst of rollouts of uneven size through the continuous-batching engine.
* ``image``    one drawn frame: a step, the particles splatted into the density volume, the ray march.
* ``voxel``    a triangle mesh turned into a voxel mask.
* ``product``  one operator product of the eigen-solve (Chebyshev recurrence on a block of vectors).
* ``tensor``   the advection tensor of a domain from its eigenbasis.

Bases are built here from analytic modes of the box (discretely divergence-free products of sines and
cosines, zero on faces of solid voxels) and a random energy-preserving advection tensor of the magnitude
the real one has, so a case needs no eigen-solve; they depend on the domain only, as a basis loaded from
a file does, and everything else is made from the seed.
"""

import ctypes as ct
import math

import numpy as np
import torch

from parallelspectralfluids3d_b200 import _lib as L
from parallelspectralfluids3d_b200 import basis as host_basis
from parallelspectralfluids3d_b200 import precompute, voxel
from parallelspectralfluids3d_b200._lib_pre import WedgeDesc
from parallelspectralfluids3d_b200.batch import Batch
from parallelspectralfluids3d_b200.domain import box_domain, sphere_obstacle_domain
from parallelspectralfluids3d_b200.engine import Engine
from parallelspectralfluids3d_b200.fixture import Basis
from parallelspectralfluids3d_b200.solver import Context
from parallelspectralfluids3d_b200.volume import Volume, make_view

F64 = torch.float64


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # The interactive loop at its smallest: one step of the 16^3 box, the particles read for drawing.
        dict(name="frame_box16_n64", kind="rollout", dims="16,16,16", radius=0.0, modes=64, particles=4096,
             steps=1, reset=False, rk=4, speed=1.0, force=0.0, viscosity=0.0, life=0.0),
        # The benchmark's default workload as a rollout: obstacle, forcing, RK4.
        dict(name="rollout_sphere32_n128", kind="rollout", dims="32,32,32", radius=8.0, modes=128,
             particles=262144, steps=100, reset=True, rk=4, speed=1.0, force=0.1, viscosity=0.0, life=0.0),
        # Reference defaults (forward Euler, lifetimes with respawn, viscosity, gravity) on a ragged grid.
        dict(name="rollout_ragged_rk1", kind="rollout", dims="27,33,21", radius=0.0, modes=93,
             particles=100003, steps=60, reset=True, rk=1, speed=10.0, force=0.05, viscosity=0.01, life=60.0),
        # The largest single instance: 48^3 channel, N = 256, a million particles.
        dict(name="rollout_channel48_n256", kind="rollout", dims="48,48,48", radius=0.0, modes=256,
             particles=1 << 20, steps=60, reset=True, rk=4, speed=10.0, force=0.0, viscosity=0.0, life=0.0),
        # Serving's largest basis: 64 instances of N = 384, few particles (coefficient-bound).
        dict(name="batch64_channel64_n384", kind="batch", domains="64,32,32/0", modes=384, slots=64,
             particles=16384, steps=50, rk=4, speed=1.0, uneven=False),
        # The batching configuration: 512 instances of uneven N over three domains.
        dict(name="batch512_mixed", kind="batch", domains="32,32,32/0 40,40,40/10 64,32,32/0", modes=256,
             slots=171, particles=16384, steps=40, rk=4, speed=1.0, uneven=True),
        # Particle-heavy batch: 32 instances of the default workload (tracer-bound).
        dict(name="batch32_sphere32_p262144", kind="batch", domains="32,32,32/8", modes=128, slots=32,
             particles=262144, steps=60, rk=4, speed=30.0, uneven=False),
        # A burst of requests to the serving engine, every result collected.
        dict(name="serve_burst24", kind="serve", domains="32,32,32/0 32,32,32/8", modes=192, requests=24,
             min_particles=10000, max_particles=300000, min_steps=50, max_steps=200),
        # One drawn frame at 720p.
        dict(name="image_sphere32_720p", kind="image", dims="32,32,32", radius=8.0, modes=128,
             particles=262144, rk=4, speed=10.0, res=256, width=1280, height=720),
        # Loading a model: mesh to voxel mask.
        dict(name="voxel_sphere_160", kind="voxel", subdivisions=6, voxels=160, mode=0),
        # Precompute: one degree of the eigen-solve's filter, and a tensor.
        dict(name="product_sphere32_c160", kind="product", dims="32,32,32", radius=8.0, columns=160),
        dict(name="tensor_box16_n128", kind="tensor", dims="16,16,16", radius=0.0, modes=128),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dims(rng, lo, hi):
    return ",".join(str(rng.randint(lo, hi)) for _ in range(3))


def draw(rng):
    kind = rng.choice(["rollout", "rollout", "rollout", "batch", "batch", "batch", "serve", "image", "voxel",
                       "product", "tensor"])
    rk = rng.choice([1, 4, 4])
    if kind == "rollout":
        n = _log(rng, 12, 44)
        dims = _dims(rng, max(10, int(0.7 * n)), n)
        reset = rng.random() < 0.75
        return dict(kind=kind, dims=dims, radius=rng.choice([0.0, 0.2 * min(map(int, dims.split(",")))]),
                    modes=_log(rng, 16, 256), particles=_log(rng, 1000, 600000),
                    steps=_log(rng, 8, 100) if reset else rng.randint(1, 3), reset=reset, rk=rk,
                    speed=rng.choice([1.0, 10.0, 30.0]), force=rng.choice([0.0, 0.05]) if reset else 0.0,
                    viscosity=0.0, life=0.0)
    if kind == "batch":
        doms = " ".join(f"{_dims(rng, 16, 36)}/{rng.choice([0, 5])}" for _ in range(rng.choice([1, 1, 2])))
        return dict(kind=kind, domains=doms, modes=_log(rng, 32, 300), slots=rng.randint(4, 80),
                    particles=_log(rng, 2000, 60000), steps=rng.randint(10, 50), rk=rk,
                    speed=rng.choice([1.0, 10.0, 30.0]), uneven=rng.random() < 0.5)
    if kind == "serve":
        return dict(kind=kind, domains=f"{_dims(rng, 20, 36)}/0", modes=_log(rng, 64, 224),
                    requests=rng.randint(8, 24), min_particles=3000, max_particles=_log(rng, 20000, 200000),
                    min_steps=20, max_steps=rng.randint(60, 160))
    if kind == "image":
        return dict(kind=kind, dims=_dims(rng, 20, 40), radius=0.0, modes=_log(rng, 32, 128),
                    particles=_log(rng, 20000, 400000), rk=rk, speed=10.0, res=rng.choice([96, 128, 160, 256]),
                    width=rng.randint(320, 1280), height=rng.randint(200, 720))
    if kind == "voxel":
        return dict(kind=kind, subdivisions=rng.choice([4, 5, 6]), voxels=rng.randint(40, 200),
                    mode=rng.choice([0, 1]))
    if kind == "product":
        return dict(kind=kind, dims=_dims(rng, 16, 34), radius=rng.choice([0.0, 5.0]), columns=_log(rng, 24, 240))
    return dict(kind=kind, dims=_dims(rng, 10, 18), radius=0.0, modes=_log(rng, 24, 160))


# ------------------------------------------------------------- domain, basis
_bases = {}


def _domain(dims, radius):
    dims = tuple(int(d) for d in dims.split(","))
    return (sphere_obstacle_domain(dims, radius) if radius > 0 else box_domain(dims)).build()


def _basis(dims, radius, modes):
    """A Basis of the domain with analytic modes; kept for the process, as a loaded file is."""
    key = (dims, float(radius), int(modes))
    if key in _bases:
        return _bases[key]
    dom = _domain(dims, radius)
    n = np.array(dom.dims)
    # Wave vectors by increasing discrete eigenvalue; one or two divergence-free polarisations each.
    top = [min(int(d) - 1, 12) for d in n]
    found = []
    for a in range(top[0] + 1):
        for b in range(top[1] + 1):
            for c in range(top[2] + 1):
                k = np.array([2.0 * math.sin(math.pi * m / (2.0 * d)) for m, d in zip((a, b, c), n)])
                zero = [m == 0 for m in (a, b, c)]
                if sum(zero) >= 2:
                    continue
                if any(zero):
                    p, q = [i for i in range(3) if not zero[i]]
                    v = np.zeros(3)
                    v[p], v[q] = k[q], -k[p]
                    found.append((float(k @ k), (a, b, c), v))
                else:
                    e = np.cross(k, [1.0, 0.0, 0.0])
                    for v in (e, np.cross(k, e)):
                        found.append((float(k @ k), (a, b, c), v))
    found.sort(key=lambda m: (m[0], m[1]))
    found = found[:modes]
    if len(found) < modes:
        raise ValueError("grid too small for the mode count")
    I = dom.interior_faces
    ax = torch.from_numpy(dom.face_axis[I].astype(np.int64)).cuda()
    xyz = torch.from_numpy(dom.face_xyz[I]).cuda()
    wave = torch.tensor([m[1] for m in found], dtype=F64, device="cuda")
    pol = torch.tensor(np.array([m[2] for m in found]), dtype=F64, device="cuda")
    phi = pol[:, ax].T.contiguous()  # [face][mode]: the component along the face's axis
    for d in range(3):
        normal = (ax == d).unsqueeze(1)
        at = torch.where(normal[:, 0], xyz[:, d].to(F64), xyz[:, d].to(F64) + 0.5)
        arg = at.unsqueeze(1) * wave[:, d] * (math.pi / float(n[d]))
        phi *= torch.where(normal, torch.sin(arg), torch.cos(arg))
        del arg
    phi /= torch.linalg.vector_norm(phi, dim=0)
    # The tracer reads z-faces with a minus sign (interior faces; +1 on x and y).
    phi *= torch.where(ax == 2, -1.0, 1.0).to(F64).unsqueeze(1)
    g = torch.Generator(device="cuda")
    g.manual_seed(977)
    R = torch.randn((modes, modes, modes), generator=g, dtype=F64, device="cuda")
    C = (R - R.transpose(0, 1)) * (1e-3 / math.sqrt(2.0 * modes))  # w . dw = 0
    b = Basis(dom.dims, dom.h, dom.aabb_min, dom.aabb_max, I.astype(np.int32),
              np.array([m[0] for m in found]) / (2.0 * dom.h), np.zeros(modes), phi.cpu().numpy(),
              C.contiguous().cpu().numpy(), dom.sign_bits, dom.inside.ravel().astype(np.uint8), name=dom.name)
    _bases[key] = b
    return b


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return g


def _coefficients(g, modes, speed):
    w = torch.randn(modes, generator=g, dtype=F64, device="cuda")
    return (w * (speed / torch.linalg.vector_norm(w))).cpu().numpy()


def _particles(g, b, count, life):
    """Uniform over the fluid voxels, float4; lifetimes uniform in [0, life) or endless."""
    fluid = torch.from_numpy(np.nonzero(b.inside)[0]).cuda()
    v = fluid[torch.randint(len(fluid), (count,), generator=g, device="cuda")]
    nx, ny, _ = b.dims
    cell = torch.stack([v % nx, (v // nx) % ny, v // (nx * ny)], 1).to(F64)
    p = (cell + torch.rand((count, 3), generator=g, dtype=F64, device="cuda")) * b.h
    p = (p + torch.from_numpy(b.aabb_min.astype(np.float64)).cuda()).float()
    t = torch.floor(torch.rand(count, generator=g, device="cuda") * life) if life > 0 else \
        torch.full((count,), math.inf, device="cuda")
    out = torch.empty((count, 4), dtype=torch.float32, pin_memory=True)
    out.copy_(torch.cat([p, t.unsqueeze(1)], 1))
    return out.numpy()


def _pinned(shape, dtype):
    return torch.empty(shape, dtype=dtype, pin_memory=True).numpy()


def _flags(force):
    return L.PSF_FLAG_RENORM | (L.PSF_FLAG_FORCING if force else 0)


DT = 0.005


def _forcing(modes, force):
    f = np.zeros(modes)
    f[0] = force / DT
    return f


# ------------------------------------------------------------------ prepare
def _rollout_inputs(case, seed):
    b = _basis(case["dims"], case["radius"], case["modes"])
    g = _generator(seed)
    w0 = _coefficients(g, b.n_modes, case["speed"])
    return b, w0, _particles(g, b, case["particles"], case.get("life", 0.0))


def _rollout(case, seed):
    b, w0, parts = _rollout_inputs(case, seed)
    force = case.get("force", 0.0)
    params = L.make_params(dt=DT, integrator=case["rk"], flags=_flags(force), viscosity=case.get("viscosity", 0.0),
                           lifetime=case.get("life", 0.0) or math.inf, seed=seed & 0xFFFF)
    ctx = Context(b, params, forcing=_forcing(b.n_modes, force))
    ctx.set_state(w0)
    ctx.set_particles(parts)
    return dict(kind="rollout", ctx=ctx, w0=w0, parts=parts, steps=case.get("steps", 1),
                reset=case.get("reset", False), w=_pinned(b.n_modes, F64), p=_pinned(parts.shape, torch.float32))


def _domains(case):
    return [(d.split("/")[0], float(d.split("/")[1])) for d in case["domains"].split()]


def _batch_mix(case):
    """(basis index, slot, modes) of every instance, slot by slot over the domains; a property of the case."""
    mix = np.random.default_rng(case["slots"] * 1000 + case["modes"])
    n = case["modes"]
    return [(i, s, max(8, int(n * mix.choice([0.125, 0.25, 0.375, 0.5, 0.75, 1.0]))) if case["uneven"] else n)
            for s in range(case["slots"]) for i in range(len(_domains(case)))]


def _batch_inputs(case, seed):
    """One entry per instance: (basis index, slot, modes, w0, particles)."""
    bases = [_basis(d, r, case["modes"]) for d, r in _domains(case)]
    g = _generator(seed)
    return bases, [(i, s, n, _coefficients(g, n, case["speed"]), _particles(g, bases[i], case["particles"], 0.0))
                   for i, s, n in _batch_mix(case)]


def _batch(case, seed):
    bases, inst = _batch_inputs(case, seed)
    bt = Batch(bases, case["slots"], case["particles"])
    params = L.make_params(dt=DT, integrator=case["rk"], flags=_flags(0.0), precision=L.PSF_PRECISION_BF16X2)
    status = bt.set_instances([dict(basis=i, slot=s, n_modes=n, w0=w0, params=params, particles=p)
                               for i, s, n, w0, p in inst])
    if status.any():
        raise RuntimeError(f"placement failed: {status}")
    n = len(inst)
    w = _pinned(sum(x[2] for x in inst), F64)
    p = _pinned((n * case["particles"], 4), torch.float32)
    wp, pp, at = (ct.c_void_p * n)(), (ct.c_void_p * n)(), 0
    for k, x in enumerate(inst):
        wp[k] = w[at:].ctypes.data
        pp[k] = p[k * case["particles"]:].ctypes.data
        at += x[2]
    return dict(kind="batch", bt=bt, steps=case["steps"], n=n, basis=np.array([x[0] for x in inst], np.int32),
                slot=np.array([x[1] for x in inst], np.int32), wp=wp, pp=pp, w=w, p=p)


def _serve_mix(case):
    """(basis index, modes, steps, particles) of every request; a property of the case."""
    mix = np.random.default_rng(case["requests"] * 1000 + case["modes"])
    out = []
    for k in range(case["requests"]):
        n = int(mix.integers(max(16, case["modes"] // 3), case["modes"] + 1))
        steps = int(mix.integers(case["min_steps"], case["max_steps"] + 1))
        P = int(math.exp(mix.uniform(math.log(case["min_particles"]), math.log(case["max_particles"]))))
        out.append((k % len(_domains(case)), n, steps, P))
    return out


def _serve_inputs(case, seed):
    bases = [_basis(d, r, case["modes"]) for d, r in _domains(case)]
    g = _generator(seed)
    return bases, [(i, steps, _coefficients(g, n, 1.0), _particles(g, bases[i], P, 0.0))
                   for i, n, steps, P in _serve_mix(case)]


def _serve(case, seed):
    bases, reqs = _serve_inputs(case, seed)
    slots = -(-case["requests"] // len(bases))
    eng = Engine(bases, slots, case["max_particles"], chunk_steps=16)
    params = L.make_params(dt=DT, flags=_flags(0.0), precision=L.PSF_PRECISION_BF16X2)
    return dict(kind="serve", eng=eng, reqs=reqs, params=params)


def _image(case, seed):
    s = _rollout(case, seed)
    eye = np.random.default_rng(seed).normal(size=3)
    eye = eye / np.linalg.norm(eye) * 1.7
    s.update(kind="image", vol=Volume(case["res"]),
             view=make_view(case["width"], case["height"], eye, light=(1.0, 2.0, 1.5)))
    return s


def _voxel(case, seed):
    v, t = voxel.icosphere(case["subdivisions"], 0.5, (0.0, 0.0, 0.0))
    rng = np.random.default_rng(seed)
    k = rng.normal(size=(4, 3)) * 4.0
    bump = 1.0 + 0.05 * np.sin(v.astype(np.float64) @ k.T + rng.uniform(0, 6.28, 4)).sum(1)
    v = v * bump[:, None]
    v = (0.1 + 0.9 * (v - v.min(0)) / (v.max(0) - v.min(0))).astype(np.float32)  # the grid starts at the origin
    res = 1.0 / case["voxels"]
    dims, _, _ = voxel.grid(v, res, case["mode"])
    vx = voxel.Voxelizer(len(v), len(t), int(np.prod(dims)))
    return dict(kind="voxel", vx=vx, v=v, t=t, res=res, mode=case["mode"])


_operators = {}


def _operator(case):
    key = (case["dims"], case["radius"])
    if key not in _operators:
        _operators[key] = host_basis.laplacian_interior(_domain(*key)).tocsr()
    return _operators[key]


def _blocks(case, seed):
    K = _operator(case)
    g = _generator(seed)
    ld = case["columns"] + (case["columns"] & 1)
    return K, [torch.randn((K.shape[0], ld), generator=g, dtype=F64, device="cuda") for _ in range(2)]


CHEB = dict(alpha=0.7, beta=-1.1, gamma=-0.4)


def _product(case, seed):
    K, (Y, X) = _blocks(case, seed)
    return dict(kind="product", A=precompute.DeviceCSR(K, Y.device), Y=Y, X=X, out=torch.empty_like(Y))


_wedges = {}


def _tensor_inputs(case, seed):
    key = (case["dims"], case["radius"])
    if key not in _wedges:
        dom = _domain(*key)
        uniq, faces, S = precompute.wedge_data(dom)
        _wedges[key] = (len(uniq), len(dom.interior_faces), torch.from_numpy(faces).cuda(),
                        torch.from_numpy(np.ascontiguousarray(S)).cuda())
    E, F, faces, S = _wedges[key]
    N = case["modes"]
    ldn = (N + 127) // 128 * 128
    g = _generator(seed)
    phi = torch.zeros((F + 1, ldn), dtype=F64, device="cuda")
    phi[:F, :N] = torch.randn((F, N), generator=g, dtype=F64, device="cuda") / math.sqrt(F)
    psi = torch.zeros((E, ldn), dtype=F64, device="cuda")
    psi[:, :N] = torch.randn((E, N), generator=g, dtype=F64, device="cuda") / math.sqrt(E)
    lam = 0.1 + torch.rand(N, generator=g, dtype=F64, device="cuda")
    return E, F, N, ldn, faces, S, phi, psi, lam


def _tensor(case, seed):
    E, F, N, ldn, faces, S, phi, psi, lam = _tensor_inputs(case, seed)
    desc = WedgeDesc(E, N, ldn, faces.data_ptr(), S.data_ptr(), psi.data_ptr(), phi.data_ptr(), F, lam.data_ptr())
    lib = L.load()
    kb = min(N, 64)
    need = ct.c_int64()
    L.check(lib.psf_pre_advection_workspace(ct.byref(desc), kb, ct.byref(need)))
    return dict(kind="tensor", lib=lib, desc=desc, kb=kb, need=need.value, keep=(faces, S, phi, psi, lam),
                ws=torch.empty((need.value + 255) // 8, dtype=F64, device="cuda"),
                C=torch.empty((N, N, N), dtype=F64, device="cuda"))


def prepare(case, seed):
    return {"rollout": _rollout, "batch": _batch, "serve": _serve, "image": _image, "voxel": _voxel,
            "product": _product, "tensor": _tensor}[case["kind"]](case, seed)


# ---------------------------------------------------------------------- run
def run(s):
    kind = s["kind"]
    if kind == "rollout":
        ctx = s["ctx"]
        if s["reset"]:
            ctx.set_state(s["w0"])
            ctx.set_particles(s["parts"])
        ctx.step(s["steps"])
        return ctx.get_state(s["w"]), ctx.get_particles(s["p"])
    if kind == "batch":
        bt = s["bt"]
        bt.step(s["steps"])
        L.check(bt.lib.psf_batch_read_instances(bt.handle, s["n"], L.ptr(s["basis"], ct.c_int32),
                                                L.ptr(s["slot"], ct.c_int32), s["wp"], s["pp"]))
        return s["w"], s["p"]
    if kind == "serve":
        eng = s["eng"]
        ids = [eng.submit(i, w0, steps, s["params"], particles=p) for i, steps, w0, p in s["reqs"]]
        out = []
        for rid in ids:
            if not eng.wait(rid):
                raise RuntimeError("a request did not finish")
            out.extend(eng.collect(rid)[:2])
        return out
    if kind == "image":
        s["ctx"].step(1)
        s["vol"].splat_context(s["ctx"])
        return s["vol"].render(s["view"])
    if kind == "voxel":
        return s["vx"].run(s["v"], s["t"], s["res"], s["mode"])[0]
    if kind == "product":
        return precompute.csr_apply(s["A"], s["Y"], s["out"], X=s["X"], **CHEB)
    L.check(s["lib"].psf_pre_advection_tensor(ct.byref(s["desc"]), s["kb"], s["ws"].data_ptr(), s["need"],
                                              s["C"].data_ptr(),
                                              ct.c_void_p(torch.cuda.current_stream().cuda_stream)))
    return s["C"]


# --------------------------------------------------------------------- work
STAGE_FLOPS = 75  # one trilinear velocity evaluation of three staggered components


def _faces(dims):
    x, y, z = (int(d) for d in dims.split(","))
    return (x - 1) * y * z + x * (y - 1) * z + x * y * (z - 1)


def _step_work(dims, modes, particles, rk, share=1.0):
    """Bytes and operations of one step of one instance that has `share` of its basis' one reading."""
    f = _faces(dims)
    return (share * 4.0 * (modes ** 3 + f * modes) + 8.0 * f + 32.0 * particles,
            2.0 * modes ** 3 + 2.0 * f * modes + particles * STAGE_FLOPS * rk)


def work(case):
    kind = case["kind"]
    if kind in ("rollout", "image"):
        by, fl = _step_work(case["dims"], case["modes"], case["particles"], case["rk"])
        if kind == "rollout":
            io = 16.0 * case["particles"] * (2 if case["reset"] else 1)
            return dict(bytes=by * case["steps"] + io, flops=fl * case["steps"])
        cells, pixels = case["res"] ** 3, case["width"] * case["height"]
        return dict(bytes=by + 16.0 * case["particles"] + 2.0 * cells + 16.0 * pixels, flops=fl + pixels * 256 * 40.0)
    if kind == "batch":
        by = fl = 0.0
        mix, doms = _batch_mix(case), _domains(case)
        for i, _, n in mix:
            by += _step_work(doms[i][0], case["modes"], case["particles"], case["rk"], 1.0 / case["slots"])[0]
            fl += _step_work(doms[i][0], n, case["particles"], case["rk"])[1]
        return dict(bytes=by * case["steps"] + 16.0 * len(mix) * case["particles"], flops=fl * case["steps"])
    if kind == "serve":
        doms = _domains(case)
        by = fl = 0.0
        for i, n, steps, P in _serve_mix(case):
            b, f = _step_work(doms[i][0], n, P, 4, len(doms) / case["requests"])
            by += b * steps + 32.0 * P
            fl += f * steps
        return dict(bytes=by, flops=fl)
    if kind == "voxel":
        t = 20 * 4 ** case["subdivisions"]
        return dict(bytes=float(case["voxels"] ** 3 + 18 * t), flops=60.0 * t)
    if kind == "product":
        f = _faces(case["dims"])
        return dict(bytes=24.0 * f * case["columns"] + 156.0 * f, flops=30.0 * f * case["columns"])
    x, y, z = (int(d) for d in case["dims"].split(","))
    e, n = 3.0 * x * y * z, case["modes"]
    return dict(bytes=8.0 * (n ** 3 + 2 * e * n + 64 * e), flops=2.0 * e * n ** 3)


# -------------------------------------------------------------------- exact
def _hash(seed, step, idx, k):
    """The respawn generator: SplitMix64's output function over (seed, step, particle, draw)."""
    with np.errstate(over="ignore"):
        u = np.uint64
        x = u(seed) ^ (u(step) * u(0x9E3779B97F4A7C15)) ^ (idx.astype(u) << u(32)) ^ (u(k) * u(0xD1B54A32D192ED03))
        x ^= x >> u(30)
        x *= u(0xBF58476D1CE4E5B9)
        x ^= x >> u(27)
        x *= u(0x94D049BB133111EB)
        x ^= x >> u(31)
    return (x >> u(32)).astype(np.int64)


class _Exact:
    """Instances of one basis stepped in 64 bits: w [B][N], p [B][P][4]."""

    def __init__(self, b, rk, force=0.0, viscosity=0.0, life=0.0, seed=0):
        self.b, self.rk, self.viscosity, self.life, self.seed = b, rk, viscosity, life, seed
        self.C = torch.from_numpy(b.C).cuda()
        self.phi = torch.from_numpy(b.phi).cuda()
        self.lam = torch.from_numpy(b.lam).cuda()
        self.force = torch.from_numpy(_forcing(b.n_modes, force)).cuda()
        nx, ny, nz = b.dims
        self.shape = [(nz, ny, nx + 1), (nz, ny + 1, nx), (nz + 1, ny, nx)]
        sizes = [int(np.prod(s)) for s in self.shape]
        face = torch.from_numpy(b.active_faces.astype(np.int64)).cuda()
        nz_f, ny_f = sizes[2], sizes[1]  # reference numbering: z-faces, y-faces, x-faces
        self.where = [face >= nz_f + ny_f, (face >= nz_f) & (face < nz_f + ny_f), face < nz_f]
        first = [nz_f + ny_f, nz_f, 0]
        self.at = [face[m] - o for m, o in zip(self.where, first)]
        self.sizes = sizes
        self.mn = torch.from_numpy(b.aabb_min.astype(np.float64)).cuda()
        self.mx = torch.from_numpy(b.aabb_max.astype(np.float64)).cuda()

    def coefficients(self, w, live):
        N = self.b.n_modes
        Y = (self.C.reshape(N * N, N) @ w.T).reshape(N, N, -1)
        dw = torch.einsum("ba,kab->bk", w, Y) * live
        w1 = w + DT * dw
        w1 = w1 * torch.sqrt((w * w).sum(1, keepdim=True) / (w1 * w1).sum(1, keepdim=True))
        return (w1 * torch.exp(self.viscosity * self.lam * DT) + DT * self.force) * live

    def fields(self, w):
        u = w @ self.phi.T
        out = []
        for d in range(3):
            f = torch.zeros((w.shape[0], self.sizes[d]), dtype=F64, device="cuda")
            f[:, self.at[d]] = u[:, self.where[d]] * (-1.0 if d == 2 else 1.0)
            out.append(f.reshape(-1))
        return out

    def velocity(self, fields, q, base):
        gw = (q - self.mn) / self.b.h
        n = torch.tensor(self.b.dims, device="cuda")
        top = n - 1
        whole = torch.minimum(torch.clamp(torch.floor(gw).long(), min=0), top)
        r = torch.floor(gw - 0.5).long()
        lo = torch.minimum(torch.clamp(r, min=0), top)
        hi = torch.minimum(torch.clamp(r + 1, min=0), top)
        out = []
        for d in range(3):
            _, sy, sx = self.shape[d]
            i0 = [whole[..., a] if a == d else lo[..., a] for a in range(3)]
            i1 = [whole[..., a] + 1 if a == d else hi[..., a] for a in range(3)]
            t = [gw[..., a] - (i0[a] if a == d else lo[..., a] + 0.5) for a in range(3)]
            v = []
            for iz in (i0[2], i1[2]):
                row = []
                for ix in (i0[0], i1[0]):
                    y0, y1 = (fields[d][base[d] + (iz * sy + iy) * sx + ix] for iy in (i0[1], i1[1]))
                    row.append(y0 + t[1] * (y1 - y0))
                v.append(row[0] + t[0] * (row[1] - row[0]))
            out.append(v[0] + t[2] * (v[1] - v[0]))
        return torch.stack(out, -1)

    def trace(self, fields, p, step):
        x, life = p[..., :3], p[..., 3]
        base = [torch.arange(p.shape[0], device="cuda").unsqueeze(1) * s for s in self.sizes]
        clamp = lambda q: torch.minimum(torch.maximum(q, self.mn), self.mx)  # noqa: E731
        k1 = self.velocity(fields, x, base)
        v = k1
        if self.rk == 4:
            k2 = self.velocity(fields, clamp(x + 0.5 * DT * k1), base)
            k3 = self.velocity(fields, clamp(x + 0.5 * DT * k2), base)
            k4 = self.velocity(fields, clamp(x + DT * k3), base)
            v = (k1 + 2 * k2 + 2 * k3 + k4) / 6
        out = torch.cat([clamp(x + DT * v), (life - 1).unsqueeze(-1)], -1)
        dead = ~(life > 0)
        if self.life > 0 and bool(dead.any()):
            idx = np.arange(p.shape[1])
            r = [torch.from_numpy((_hash(self.seed, step, idx, k) % 1024) / 1024.0).cuda() for k in (1, 2, 3)]
            centre = float(self.mn[2] + 0.5 * (self.mx[2] - self.mn[2]))
            new = torch.stack([(r[0] - 0.5) * 0.25, torch.full_like(r[0], float(self.mn[1]) + float(np.float32(0.2))),
                               (r[2] - 0.5) * 0.25 - centre, self.life * r[1]], -1)
            out = torch.where(dead.unsqueeze(-1), new.unsqueeze(0), out)
        return out

    def run(self, w, p, steps, n_modes=None):
        live = torch.ones_like(w)
        if n_modes is not None:
            for i, n in enumerate(n_modes):
                live[i, n:] = 0
        for step in range(steps):
            w = self.coefficients(w, live)
            p = self.trace(self.fields(w), p, step)
        return w, p


def exact(case, seed):
    kind = case["kind"]
    if kind == "rollout":
        b, w0, parts = _rollout_inputs(case, seed)
        ex = _Exact(b, case["rk"], case["force"], case["viscosity"], case["life"], seed & 0xFFFF)
        w, p = ex.run(torch.from_numpy(w0).cuda()[None], torch.from_numpy(parts).cuda().double()[None], case["steps"])
        return w[0], p[0]
    if kind == "batch":
        bases, inst = _batch_inputs(case, seed)
        if len(inst) * case["particles"] * case["steps"] > 6e8:  # too long: over about 20 seconds
            return None
        wo, po = [None] * len(inst), [None] * len(inst)
        for i, b in enumerate(bases):
            ex = _Exact(b, case["rk"])
            mine = [k for k, x in enumerate(inst) if x[0] == i]
            for at in range(0, len(mine), 32):
                ks = mine[at:at + 32]
                w = torch.zeros((len(ks), b.n_modes), dtype=F64, device="cuda")
                for r, k in enumerate(ks):
                    w[r, :inst[k][2]] = torch.from_numpy(inst[k][3]).cuda()
                p = torch.stack([torch.from_numpy(inst[k][4]).cuda().double() for k in ks])
                w, p = ex.run(w, p, case["steps"], [inst[k][2] for k in ks])
                for r, k in enumerate(ks):
                    wo[k], po[k] = w[r, :inst[k][2]], p[r]
        return torch.cat(wo), torch.cat(po)
    if kind == "serve":
        bases, reqs = _serve_inputs(case, seed)
        ex = [_Exact(b, 4) for b in bases]
        out = []
        for i, steps, w0, parts in reqs:
            w = torch.zeros((1, bases[i].n_modes), dtype=F64, device="cuda")
            w[0, :len(w0)] = torch.from_numpy(w0).cuda()
            w, p = ex[i].run(w, torch.from_numpy(parts).cuda().double()[None], steps, [len(w0)])
            out += [w[0, :len(w0)], p[0]]
        return out
    if kind == "product":
        K, (Y, X) = _blocks(case, seed)
        A = torch.sparse_csr_tensor(torch.from_numpy(K.indptr.astype(np.int64)).cuda(),
                                    torch.from_numpy(K.indices.astype(np.int64)).cuda(),
                                    torch.from_numpy(K.data).cuda(), size=K.shape)
        return CHEB["alpha"] * (A @ Y) + CHEB["beta"] * Y + CHEB["gamma"] * X
    if kind == "tensor":
        E, F, N, _, faces, S, phi, psi, lam = _tensor_inputs(case, seed)
        pf = phi[faces.long(), :N]  # [E][8][N]; unused slots are the zero row
        Spf = torch.einsum("efg,efk->egk", S, pf)
        C = torch.empty((N, N, N), dtype=F64, device="cuda")
        for k in range(N):
            C[k] = psi[:, :N].T @ torch.einsum("eg,egj->ej", Spf[:, :, k], pf) / lam[k]
        return C
    # Voxel masks are whole bytes; an image in 64 bits is 10^9 trilinear shadow samples (minutes).
    return None
