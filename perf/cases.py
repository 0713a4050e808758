"""The workloads whose speed is followed: what a program that uses this package
has it do, over the sizes it is used at.

``listed()`` names them, ``draw(rng)`` gives another one of the same ranges,
``prepare(case, seed)`` makes what such a program holds before the call,
``run(state)`` is one pass through the package's public entry points,
``work(case)`` what that pass cannot do without, and ``exact(case, seed)`` its
results as plain torch computes them in 64 bits.

Kinds of pass:

* ``force``  one particle-mesh force evaluation on particles held on the GPU
* ``run``    one realization: particles loaded, the time loop, the snapshot
* ``batch``  several realizations of uneven boxes and lengths in one graph
* ``pk``     the power spectrum of the particles' density
* ``fof``    friends-of-friends halos of a snapshot
* ``lpt``    the 2LPT initial conditions of one seed, into host memory
* ``net``    the coarse force with the conv net's correction
* ``train``  one optimiser step of that net
"""
import ctypes
import math
import os
import tempfile

import numpy as np
import torch

from cola_halo_b200 import _lib
from cola_halo_b200.batch import Batch
from cola_halo_b200.bbks import write_bbks_table
from cola_halo_b200.halos import HALO_DTYPE
from cola_halo_b200.learned import ConvNet, copy_particles
from cola_halo_b200.schedule import Schedule
from cola_halo_b200.sim import Simulation
from cola_halo_b200.types import PARTICLE_DTYPE, Particles

OMEGA_M = 0.273
DEV = "cuda"
MESHES = (16, 32, 48, 64, 96, 128, 144, 192, 256, 384, 512, 768, 1024)


# ------------------------------------------------------------------ cases

def _case(kind, nc, ngrid, boxsize, **more):
    return dict(kind=kind, nc=nc, ngrid=ngrid, boxsize=boxsize, **more)


def _force(nc, ngrid, boxsize, stage="late", gradient=0, laplacian=0, deconvolve=0, knots=0):
    return _case("force", nc, ngrid, boxsize, stage=stage, gradient=gradient,
                 laplacian=laplacian, deconvolve=deconvolve, knots=knots)


def listed():
    return [
        # a small test box, called from a user's own loop: launches and latency
        dict(_force(32, 96, 100.0), name="force_32p_96m"),
        # a particle count that is no power of two on a mesh that is no
        # multiple of it
        dict(_force(100, 256, 250.0), name="force_100p_256m"),
        # the coarse mesh of the learned correction: the CIC window divided
        # out twice and a transfer function of 32 knots
        dict(_force(128, 128, 300.0, deconvolve=2, knots=32), name="force_128p_128m_filter"),
        # the largest mesh: 512^3 particles, factor 2, at their first step
        dict(_force(512, 1024, 1200.0, stage="ics"), name="force_512p_1024m"),
        # a whole small realization, z = 49 to 0
        dict(_case("run", 64, 192, 200.0, steps=10), name="run_64p_192m"),
        # a whole realization at the headline size
        dict(_case("run", 256, 768, 600.0, steps=10), name="run_256p_768m"),
        # production of many realizations: uneven boxes and step counts
        dict(_case("batch", 128, 384, 250.0, nreal=4, steps=5), name="batch_4x128p_384m"),
        # measuring a realization
        dict(_case("pk", 256, 512, 600.0), name="pk_256p_512m"),
        # the halo catalogue of a late snapshot
        dict(_case("fof", 256, 0, 600.0, linking=0.2), name="fof_256p"),
        # initial conditions of one seed
        dict(_case("lpt", 128, 0, 300.0), name="lpt_128p"),
        # the learned correction in a run, and its training
        dict(_case("net", 128, 128, 300.0), name="net_128p_128m"),
        dict(_case("train", 128, 128, 300.0, factor=3), name="train_128p_128m"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("force", "force", "force", "run", "batch", "pk", "fof", "lpt", "net",
                       "train"))
    per = rng.uniform(1.5, 3.5)          # mean particle spacing, Mpc/h
    if kind == "force":
        nc = _log_int(rng, 20, 400)
        ngrid = rng.choice([m for m in MESHES if nc <= m <= 4 * nc])
        grad = rng.choice((0, 0, 2, 4))
        return _force(nc, ngrid, nc * per, stage=rng.choice(("ics", "late", "late")),
                      gradient=grad, laplacian=rng.choice((0, 1)) if grad else 0,
                      deconvolve=rng.choice((0, 0, 2)) if ngrid <= nc * 1.25 or grad else 0,
                      knots=rng.choice((0, 0, 16, 32)))
    if kind == "run":
        nc, f = rng.choice(((32, 2), (32, 3), (48, 3), (64, 2), (64, 3), (96, 2), (128, 2),
                            (128, 3), (171, 3), (192, 2)))
        ngrid = max(m for m in MESHES if m <= f * nc)
        return _case("run", nc, ngrid, nc * per, steps=rng.randint(2, 10))
    if kind == "batch":
        nc, f = rng.choice(((32, 2), (32, 3), (48, 2), (64, 3), (96, 2), (128, 2), (128, 3)))
        return _case("batch", nc, f * nc, nc * per, nreal=rng.randint(2, 6),
                     steps=rng.randint(2, 6))
    if kind == "pk":
        nc = _log_int(rng, 24, 256)
        return _case("pk", nc, rng.choice([m for m in MESHES if nc <= m <= min(4 * nc, 768)]),
                     nc * per)
    if kind == "fof":
        return _case("fof", _log_int(rng, 40, 256), 0, rng.uniform(100.0, 700.0),
                     linking=round(rng.uniform(0.15, 0.25), 3))
    if kind == "lpt":
        nc = rng.choice((32, 48, 64, 96, 128, 144, 192))
        return _case("lpt", nc, 0, nc * per)
    n = rng.choice((32, 48, 64, 96, 128))
    nc = n - rng.choice((0, 0, 3, 7))
    if kind == "net":
        return _case("net", nc, n, nc * per)
    return _case("train", nc, n, nc * per, factor=2 if n == 96 else rng.choice((2, 3)))


# ----------------------------------------------------------------- inputs
# Particles are made in plain torch from the seed alone: second-order
# Lagrangian displacements of a BBKS density field (sigma_8 = 0.81), in the
# lattice order in which initial conditions come.  "late" particles also
# sit in halos: part of the lattice, in cubes of 4^3 to 16^3, collapsed to
# isothermal balls at 200 times the mean density.

def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) & 0x7fffffff)


def _wavenumbers(n, boxsize, dtype):
    kf = 2 * math.pi / boxsize
    k = torch.fft.fftfreq(n, 1.0 / n, device=DEV, dtype=dtype) * kf
    kz = torch.fft.rfftfreq(n, 1.0 / n, device=DEV, dtype=dtype) * kf
    return k[:, None, None], k[None, :, None], kz[None, None, :]


def _linear_power(k):
    """BBKS P(k) at z = 0; the amplitude gives sigma_8 = 0.81."""
    q = torch.clamp(k, min=1e-4) / (OMEGA_M * 0.705)
    t = torch.log1p(2.34 * q) / (2.34 * q) * (
        1 + 3.89 * q + (16.1 * q) ** 2 + (5.46 * q) ** 3 + (6.71 * q) ** 4) ** -0.25
    return 1875557.49 * torch.clamp(k, min=1e-4) ** 0.96 * t * t


def _displacements(nc, boxsize, seed):
    """(dx1, dx2): 2 x [3][nc, nc, nc] float32 displacements at D = 1."""
    g = _generator(seed)
    white = torch.fft.rfftn(torch.randn((nc,) * 3, generator=g, device=DEV))
    ks = _wavenumbers(nc, boxsize, torch.float32)
    k2 = ks[0] ** 2 + ks[1] ** 2 + ks[2] ** 2
    delta = white * torch.sqrt(_linear_power(torch.sqrt(k2)) * (nc / boxsize) ** 3)
    del white
    k2[0, 0, 0] = 1.0
    delta = delta / k2                           # delta / k^2 from here on
    delta[0, 0, 0] = 0.0
    shape = (nc,) * 3
    dx1 = [torch.fft.irfftn(1j * k * delta, s=shape) for k in ks]
    d = {}
    src = torch.zeros(shape, device=DEV)
    for a in range(3):
        d[a] = torch.fft.irfftn(ks[a] * ks[a] * delta, s=shape)
    for a, b in ((0, 1), (0, 2), (1, 2)):
        src += d[a] * d[b] - torch.fft.irfftn(ks[a] * ks[b] * delta, s=shape) ** 2
    del d, delta
    s = torch.fft.rfftn(src) / k2
    s[0, 0, 0] = 0.0
    dx2 = [torch.fft.irfftn((3.0 / 7.0) * 1j * k * s, s=shape) for k in ks]
    return dx1, dx2


def _lattice(nc, boxsize):
    q = (torch.arange(nc, device=DEV, dtype=torch.float32) + 0.5) * (boxsize / nc)
    return q[:, None, None], q[None, :, None], q[None, None, :]


def _collapse(x, boxsize, seed):
    """Cubes of the lattice collapsed in place; x: [nc, nc, nc, 3]."""
    nc = x.shape[0]
    g = _generator(seed + 77003)
    for b, share in ((16, 0.04), (8, 0.12), (4, 0.2)):
        n = nc // b
        if n == 0:
            continue
        pick = (torch.rand((n, n, n), generator=g, device=DEV) < share).nonzero()
        o = torch.arange(b, device=DEV)
        i = (pick[:, 0, None] * b + o)[:, :, None, None]
        j = (pick[:, 1, None] * b + o)[:, None, :, None]
        k = (pick[:, 2, None] * b + o)[:, None, None, :]
        block = x[i, j, k]                                   # [m, b, b, b, 3]
        centre = block.mean(dim=(1, 2, 3), keepdim=True)
        way = torch.randn(block.shape, generator=g, device=DEV)
        way /= way.norm(dim=-1, keepdim=True) + 1e-20
        radius = boxsize / nc * b * (3 / (4 * math.pi * 200)) ** (1 / 3)
        u = torch.rand(block.shape[:-1] + (1,), generator=g, device=DEV)
        x[i, j, k] = centre + radius * u * way


def _wrapped(x, boxsize):
    x = x - boxsize * torch.floor(x / boxsize)
    return torch.where(x >= boxsize, torch.zeros_like(x), x)


def _particles(nc, boxsize, seed, stage, a=0.02):
    """Reference Particle records as words: int32 [nc^3, 14] (x, dx1, dx2, v, id)."""
    n = nc ** 3
    dx1, dx2 = _displacements(nc, boxsize, seed)
    d1 = _Growth(OMEGA_M).d1(a) if stage == "ics" else 1.0
    out = torch.zeros((n, 14), dtype=torch.int32, device=DEV)
    f = out.view(torch.float32)
    q = _lattice(nc, boxsize)
    x = torch.stack([q[c] + d1 * dx1[c] + d1 * d1 * dx2[c] for c in range(3)], dim=-1)
    if stage == "late":
        _collapse(x, boxsize, seed)
    f[:, 0:3] = _wrapped(x, boxsize).view(n, 3)
    del x
    for c in range(3):
        f[:, 3 + c] = dx1[c].reshape(-1)
        f[:, 6 + c] = dx2[c].reshape(-1)
    out[:, 12] = torch.arange(1, n + 1, dtype=torch.int32, device=DEV)
    return out


def _knots(n, ngrid, seed):
    """A transfer function near 1 that rises or falls towards the mesh scale."""
    if not n:
        return None
    t = np.arange(n) / (n - 1)
    r = np.random.default_rng(seed)
    return (1 + 0.3 * r.uniform(-1, 1) * t + 0.05 * r.uniform(-1, 1, n)).astype(np.float32)


def _net_params(seed, nparams):
    """Weights of a trained net's size: live channels only, as the net keeps them."""
    r = np.random.default_rng(seed)
    p = np.zeros(nparams, dtype=np.float32)
    layer = 27 * 256 + 16
    for l, (ci, co) in enumerate(((2, 16), (16, 16), (16, 3))):
        w = np.zeros((27, 16, 16))
        w[:, :ci, :co] = r.uniform(-1, 1, (27, ci, co)) * math.sqrt(6.0 / (27 * ci))
        p[l * layer: l * layer + 27 * 256] = w.ravel()
        p[l * layer + 27 * 256: l * layer + 27 * 256 + co] = r.uniform(-0.1, 0.1, co)
    return p


def _batch_specs(case):
    """Boxes up to 1.6 times the smallest, step counts from `steps` up."""
    n = case["nreal"]
    return [dict(nc=case["nc"], ngrid=case["ngrid"],
                 boxsize=float(np.float32(case["boxsize"] * (1 + 0.6 * i / n))),
                 a_init=0.02, a_final=1.0, nsteps=case["steps"] + i, aout=1.0)
            for i in range(n)]


class _DeviceArray:
    """A float array of the library in device memory, for torch; it keeps the
    handle that owns the memory alive."""

    def __init__(self, ptr, n, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f4", "version": 3,
                                         "data": (ptr, False)}


def _force_tensors(sim):
    """The forces on the device, one tensor per component (the library's own arrays)."""
    lib = sim.lib
    x, f = (ctypes.c_void_p * 3)(), (ctypes.c_void_p * 3)()
    _lib.check(lib.cg_sim_state_ptrs(sim.h, x, f), "cg_sim_state_ptrs")
    n = lib.cg_sim_np(sim.h)
    return [torch.as_tensor(_DeviceArray(p, n, sim), device=DEV) for p in f]


def _loaded(nc, ngrid, boxsize, words, a=0.5):
    sim = Simulation(nc, ngrid, boxsize, OMEGA_M)
    torch.cuda.synchronize()
    sim.set_particles_ptr(words.data_ptr(), len(words), a, a)
    sim.move()
    sim.sync()
    return sim


def prepare(case, seed):
    kind, nc, L = case["kind"], case["nc"], float(np.float32(case["boxsize"]))
    ngrid = case["ngrid"]
    s = {"case": case, "L": L}
    if kind == "lpt":
        lib = _lib.load()
        lib.cg_dropin_set_abort(0)
        path = os.path.join(tempfile.mkdtemp(), "bbks.dat")
        write_bbks_table(path)
        lib.power_init(path.encode(), 0.02, 0.81, OMEGA_M, 1 - OMEGA_M)
        n = nc ** 3
        s["lib"], s["seed"] = lib, int(seed) % 1000003 + 1
        # the particle storage of such a program: pinned, for fast downloads
        s["host"] = torch.zeros(n * 56, dtype=torch.uint8).pin_memory()
        s["p"] = s["host"].numpy().view(PARTICLE_DTYPE)
        P = Particles()
        P.p, P.np_allocated, P.np_total, P.np_average = s["host"].data_ptr(), n, n, float(n)
        s["P"] = P
        return s
    if kind == "batch":
        specs = _batch_specs(case)
        s["specs"] = specs
        s["batch"] = Batch(specs, OMEGA_M)
        s["q"], s["snap"] = [], []
        for i, sp in enumerate(specs):
            w = _particles(nc, sp["boxsize"], seed + 1009 * i, "ics")
            torch.cuda.synchronize()
            _lib.check(_lib.load().cg_batch_set_particles(s["batch"].h, i, w.data_ptr(), len(w)),
                       "cg_batch_set_particles")
            s["q"].append(w.view(torch.float32)[:, 0:3].contiguous())
            s["snap"].append(torch.zeros((len(w), 8), dtype=torch.int32, device=DEV))
        torch.cuda.empty_cache()
        return s
    if kind == "run":
        s["words"] = _particles(nc, L, seed, "ics")
        s["sched"] = Schedule.linear(0.02, 1.0, case["steps"])
        s["snap"] = torch.zeros((nc ** 3, 8), dtype=torch.int32, device=DEV)
        s["sim"] = Simulation(nc, ngrid, L, OMEGA_M)
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        return s
    words = _particles(nc, L, seed, case.get("stage", "late"))
    if kind == "fof":
        snap = torch.zeros((len(words), 8), dtype=torch.int32, device=DEV)
        snap[:, 0:3] = words[:, 0:3]
        snap[:, 6] = words[:, 12]
        g = _generator(seed + 5)
        snap.view(torch.float32)[:, 3:6] = 300 * torch.randn((len(words), 3), generator=g,
                                                             device=DEV)
        s["snap"] = snap
        s["ll"] = float(np.float32(case["linking"] * L / nc))
        s["lib"], s["nhalo"] = _lib.load(), 0
        s["halos"] = np.zeros(len(words) // 32 + 1, dtype=HALO_DTYPE)
        torch.cuda.synchronize()
    else:
        s["sim"] = _loaded(nc, ngrid, L, words)
    if kind == "force":
        s["sim"].set_force_kernel(case["gradient"], case["laplacian"], case["deconvolve"])
        if case["knots"]:
            s["sim"].set_force_filters(_knots(case["knots"], ngrid, seed))
    if kind in ("net", "train"):
        s["net"] = ConvNet(ngrid, seed=int(seed) % 1000 + 1)
        s["net"].set_params(_net_params(seed, s["net"].nparams))
    if kind == "train":
        s["fine"] = Simulation(nc, case["factor"] * ngrid, L, OMEGA_M)
        copy_particles(s["fine"], s["sim"])
        s["fine"].sync()
    del words
    torch.cuda.empty_cache()
    return s


# --------------------------------------------------------------- the pass

def _snapshot_fields(snap, q, L):
    """Displacements from the initial positions (across the periodic faces by
    the nearest image), velocities and ids of a snapshot's records."""
    f = snap.view(torch.float32)
    d = f[:, 0:3] - q
    d -= L * torch.round(d / L)
    return {"displacement": d, "v": f[:, 3:6], "id": snap[:, 6]}


def run(s):
    kind = s["case"]["kind"]
    if kind == "force":
        s["sim"].forces()
        return _force_tensors(s["sim"])
    if kind == "run":
        sim, sched = s["sim"], s["sched"]
        sim.set_particles_ptr(s["words"].data_ptr(), len(s["words"]), sched.a_init, sched.a_init)
        for i in range(1, sched.nloop):
            _, _, avel1, apos1 = sched.times(i)
            sim.move()
            sim.forces()
            sim.kick_drift(avel1, apos1)
        sim.move()
        sim.forces()
        torch.cuda.current_stream().synchronize()   # nothing still reads the last pass's records
        _lib.check(sim.lib.cg_sim_snapshot(sim.h, sched.a_final, OMEGA_M, s["snap"].data_ptr()),
                   "cg_sim_snapshot")
        return _snapshot_fields(s["snap"], s["words"].view(torch.float32)[:, 0:3], s["L"])
    if kind == "batch":
        b = s["batch"]
        b.run()
        torch.cuda.current_stream().synchronize()   # nothing still reads the last pass's records
        out = []
        for i, sp in enumerate(s["specs"]):
            _lib.check(b.lib.cg_batch_get_snapshot(b.h, i, s["snap"][i].data_ptr()), "snapshot")
            o = _snapshot_fields(s["snap"][i], s["q"][i], sp["boxsize"])
            # kept as the rows of a float32 table of spectra
            o["pk"] = b.power_spectrum(i)[1].astype(np.float32)
            out.append(o)
        return out
    if kind == "pk":
        return [v.astype(np.float32) for v in s["sim"].power_spectrum(s["case"]["ngrid"] // 2)]
    if kind == "fof":
        lib, cat, found = s["lib"], s["halos"], ctypes.c_longlong()
        _lib.check(lib.cg_fof(s["snap"].data_ptr(), len(s["snap"]), s["L"], s["ll"], 32,
                              cat.ctypes.data, len(cat), ctypes.byref(found)), "cg_fof")
        cat[found.value: s["nhalo"]] = 0         # what is left of a longer catalogue
        s["nhalo"] = found.value
        return {"count": found.value, "nfof": cat["nfof"], "x": cat["x"], "v": cat["v"]}
    if kind == "lpt":
        lib = s["lib"]
        lib.lpt_init(s["case"]["nc"], None, 0)
        if lib.lpt_set_displacement(0.02, OMEGA_M, s["seed"], s["L"], ctypes.byref(s["P"])) != 0:
            raise RuntimeError(lib.cg_last_error().decode())
        return {k: s["p"][k] for k in ("x", "dx1", "dx2", "id")}
    if kind == "net":
        s["net"].forces(s["sim"])
        return _force_tensors(s["sim"])
    loss = s["net"].train_step(s["sim"], s["fine"], 2e-3)
    return {"loss": loss, "params": s["net"].params()}


def work(case):
    """Inputs read and outputs written once, and the arithmetic of the
    transforms, the clouds and the convolutions."""
    kind, nc, n = case["kind"], case["nc"], case["ngrid"]
    np_ = nc ** 3

    def fft(m):                              # one real 3-D transform
        return 2.5 * m ** 3 * 3 * math.log2(max(m, 2))

    def force(m):                            # one forward, three inverse, 8-cell clouds
        return 4 * fft(m) + 10 * m ** 3 + 150 * np_

    if kind == "force":
        return {"bytes": 24 * np_, "flops": force(n)}
    if kind == "run":
        return {"bytes": (56 + 32) * np_, "flops": (case["steps"] + 1) * (force(n) + 40 * np_)}
    if kind == "batch":
        specs = _batch_specs(case)
        return {"bytes": len(specs) * (56 + 32) * np_,
                "flops": sum((sp["nsteps"] + 1) * (force(n) + 40 * np_) + fft(n) + 10 * n ** 3
                             for sp in specs)}
    if kind == "pk":
        return {"bytes": 12 * np_, "flops": fft(n) + 10 * n ** 3 + 40 * np_}
    if kind == "fof":
        return {"bytes": 32 * np_, "flops": 100 * np_}
    if kind == "lpt":
        # 2 x 64-bit random numbers per mode, 202 steps per 12 of them
        return {"bytes": 56 * np_, "flops": 13 * fft(nc) + np_ * 202 / 12 * 4}
    conv = n ** 3 * 27 * 2 * (2 * 16 + 16 * 16 + 16 * 3)
    if kind == "net":
        return {"bytes": 24 * np_, "flops": force(n) + 2 * fft(n) + conv + 100 * np_}
    return {"bytes": 36 * np_, "flops": force(n) + force(case["factor"] * n) + 2 * fft(n) +
            3 * conv + 200 * np_}


# ----------------------------------------------------- results in 64 bits

class _Growth:
    """Growth factors and time coefficients of the COLA integrator
    (cola.c:73-292).  For a > 0.2 the growing mode is the integral
    H int da / (a H)^3 (Heath 1977); below, the reference's own short series
    in a^3, whose values it uses there although they differ from the growing
    mode by up to 7e-4."""

    def __init__(self, omega_m):
        self.om = float(np.float32(omega_m))
        self.node, self.weight = np.polynomial.legendre.leggauss(64)
        self.norm = self._temp(1.0)

    def _int(self, f, lo, hi):
        t = 0.5 * (hi - lo)
        return t * float(np.sum(self.weight * f(0.5 * (lo + hi) + t * self.node)))

    def _temp(self, a):
        o = self.om
        if float(np.float32(a)) > 0.2:
            def h(x):
                return np.sqrt(o / x ** 3 + 1 - o)
            # a = u^2 makes the integrand smooth at 0
            grow = 2.5 * o * float(h(a)) * self._int(
                lambda u: 2 * u / (u * u * h(u * u)) ** 3, 0.0, math.sqrt(a))
            return (1 - o) ** 1.5 * 2.4 / o * grow
        return a * (1 - o) ** 1.5 / (1.5625e10 * o ** 5) * (
            1291467969.0 * a ** 12 * (o - 1) ** 4 + 1956769650.0 * a ** 9 * (o - 1) ** 3 * o +
            8000000000.0 * a ** 3 * (o - 1) * o ** 3 + 37490640625.0 * o ** 4)

    def d1(self, a):
        return self._temp(a) / self.norm

    def omega(self, a):
        return self.om / (self.om + (1 - self.om) * a ** 3)

    def d2(self, a):
        return self.d1(a) ** 2 * (self.omega(a) / self.om) ** (-1 / 143.0)

    def q(self, a):
        return np.sqrt(self.om / a ** 3 + 1 - self.om) * a ** 3

    def kick(self, av, ax, to):
        n, g1 = -2.5, self.d1(ax)
        dda = (to ** n - av ** n) * ax / self.q(ax) / (n * ax ** (n - 1))
        q1 = 1.5 * self.om * g1
        return dda, q1, q1 * g1 * (1 + 7 / 3 * self.omega(ax) ** (1 / 143.0))

    def drift(self, ax, av, to):
        n = -2.5
        dy = 0.0
        lo = ax
        while to - lo > 1e-12:               # panels that grow with a
            hi = min(to, 1.5 * lo)
            dy += self._int(lambda a: a ** n / self.q(a), lo, hi)
            lo = hi
        return dy / av ** n, self.d1(to) - self.d1(ax), self.d2(to) - self.d2(ax)

    def velocity(self, a):
        """d(D1)/dt and d(D2)/dt in the integrator's units."""
        d = self.d1(a)
        h = math.sqrt(self.om / a ** 3 + 1 - self.om)
        dv = (6 * (1 - self.om) ** 1.5 / self.norm - 1.5 * self.om * d / a) / h
        return dv, self.q(a) * self.d2(a) / a * 2 * self.omega(a) ** (6 / 11.0)


def _corners(x, n, L):
    """The eight (cell, weight) pairs of particles x [np, 3] on an n^3 mesh."""
    t = x * (n / L)
    i = torch.floor(t)
    w = t - i
    i = i.to(torch.int64) % n
    j = (i + 1) % n
    for c in range(8):
        s = [(c >> a) & 1 for a in range(3)]
        k = [(j if s[a] else i)[:, a] for a in range(3)]
        u = [(w if s[a] else 1 - w)[:, a] for a in range(3)]
        yield (k[0] * n + k[1]) * n + k[2], u[0] * u[1] * u[2]


def _density(x, n, L, weight):
    mesh = torch.full((n ** 3,), -1.0, dtype=torch.float64, device=DEV)
    for cell, w in _corners(x, n, L):
        mesh.index_add_(0, cell, w * weight)
    return mesh.view(n, n, n)


def _indices(n):
    """Signed mode numbers, the Nyquist index at +n/2 as the reference keeps it."""
    i = torch.arange(n, device=DEV, dtype=torch.float64)
    s = torch.where(i <= n // 2, i, i - n)
    return s, s[: n // 2 + 1]


def _axis_tables(n, gradient, laplacian, deconvolve):
    s, _ = _indices(n)
    w = math.pi * s / n
    g = s
    if gradient == 2:
        g = n / (2 * math.pi) * torch.sin(2 * w)
    elif gradient == 4:
        g = n / (2 * math.pi) * (8 * torch.sin(2 * w) - torch.sin(4 * w)) / 6
    lap = (n / math.pi * torch.sin(w)) ** 2 if laplacian else s * s
    sinc = torch.where(s == 0, torch.ones_like(w), torch.sin(w) / torch.where(w == 0, 1.0, w))
    return g, lap, sinc ** (-2 * deconvolve)


def _inverse(spec, n):
    """Unnormalised c2r: complex over x and y, then half-complex over z, which
    reads no imaginary part at kz = 0 and n/2."""
    spec = torch.fft.ifft2(spec, dim=(0, 1), norm="forward")
    spec[..., 0].imag.zero_()
    spec[..., n // 2].imag.zero_()
    return torch.fft.irfft(spec, n=n, dim=2, norm="forward")


def _force_exact(x, nc, n, L, gradient=0, laplacian=0, deconvolve=0, knots=None, delta=False):
    dens = _density(x, n, L, (n / nc) ** 3)
    spec = torch.fft.rfftn(dens)
    if not delta:
        del dens
    g, lap, win = _axis_tables(n, gradient, laplacian, deconvolve)
    h = n // 2 + 1
    den = lap[:, None, None] + lap[None, :, None] + lap[None, None, :h]
    den[0, 0, 0] = 1.0
    spec *= (-1.0 / n ** 3 / (2 * math.pi / L)) / den
    spec[0, 0, 0] = 0.0
    if deconvolve:
        spec *= win[:, None, None] * win[None, :, None] * win[None, None, :h]
    if knots is not None:
        s, sz = _indices(n)
        r = torch.sqrt(s[:, None, None] ** 2 + s[None, :, None] ** 2 + sz[None, None, :] ** 2)
        r *= (len(knots) - 1) / (math.sqrt(3.0) * n / 2)
        i = torch.clamp(r.to(torch.int64), max=len(knots) - 2)
        t = torch.as_tensor(knots, dtype=torch.float64, device=DEV)
        r -= i
        spec *= t[i] * (1 - r) + t[i + 1] * r
        del r, i
    del den
    out = []
    for a in range(3):
        k = g if a < 2 else g[:h]
        mesh = _inverse(spec * (1j * k).view([-1 if b == a else 1 for b in range(3)]), n)
        mesh = mesh.reshape(-1)
        f = torch.zeros(len(x), dtype=torch.float64, device=DEV)
        for cell, w in _corners(x, n, L):
            f += mesh[cell] * w
        out.append(f)
        del mesh
    return (out, dens) if delta else out


def _power_exact(x, nc, n, L):
    nb = n // 2
    spec = torch.fft.rfftn(_density(x, n, L, (n / nc) ** 3))
    s, sz = _indices(n)
    r = torch.sqrt(s[:, None, None] ** 2 + s[None, :, None] ** 2 + sz[None, None, :] ** 2)
    w = torch.full_like(r, 2.0)
    w[..., 0] = 1.0
    w[..., n // 2] = 1.0
    b = torch.floor(r + 0.5).to(torch.int64) - 1
    use = (b >= 0) & (b < nb)
    b, w, r, p = b[use], w[use], r[use], (spec.abs() ** 2)[use]
    acc = [torch.zeros(nb, dtype=torch.float64, device=DEV).index_add_(0, b, v)
           for v in (w, w * r, w * p)]
    return (2 * math.pi / L * acc[1] / acc[0], L ** 3 / n ** 6 * acc[2] / acc[0], acc[0])


def _realization_exact(words, nc, n, L, a_init, steps, batch):
    """Displacements and velocities at a = 1 (and the final positions)."""
    f = words.view(torch.float32).double()
    q, d1, d2 = f[:, 0:3].clone(), f[:, 3:6], f[:, 6:9]
    x, v = q.clone(), torch.zeros_like(q)
    gr = _Growth(OMEGA_M)
    da = (1.0 - a_init) / steps
    ax = av = float(np.float32(a_init))
    for i in range(1, steps + 2):
        x -= L * torch.floor(x / L)
        force = torch.stack(_force_exact(x, nc, n, L), dim=1)
        to_v, to_x = a_init + (i - 0.5) * da, a_init + i * da
        # the batched loop takes the output by its place among the half
        # steps; the single run at the end of its loop
        last = i == steps + 1 or (batch and a_init + (i - 1.0) * da >= 1.0)
        dda, q1, q2 = gr.kick(av, ax, to_v)
        kicked = False
        if last and batch and a_init + (i - 1.0) * da < 1.0:
            v += (-1.5 * gr.om * force - (d1 * q1 + d2 * q2)) * dda
            av = to_v
        if last:
            dda, q1, q2 = gr.kick(av, ax, 1.0)
            dv, dv2 = gr.velocity(1.0)
            acc = -1.5 * gr.om * force - (d1 * q1 + d2 * q2)
            vel = 100.0 * (v + acc * dda + d1 * dv + d2 * dv2)
            d = x - q
            return d - L * torch.round(d / L), vel, x
        v += (-1.5 * gr.om * force - (d1 * q1 + d2 * q2)) * dda
        av = float(np.float32(to_v))
        dy, e1, e2 = gr.drift(ax, av, to_x)
        x += v * dy + (d1 * e1 + d2 * e2)
        ax = float(np.float32(to_x))


def _net_exact(x, delta, params, n, L):
    """The net's three outputs at particles x (unit feature and output scales)."""
    spec = torch.fft.rfftn(delta)
    s, sz = _indices(n)
    k2 = s[:, None, None] ** 2 + s[None, :, None] ** 2 + sz[None, None, :] ** 2
    k2[0, 0, 0] = 1.0
    spec = -spec / k2
    spec[0, 0, 0] = 0.0
    phi = torch.fft.irfftn(spec, s=(n,) * 3)
    act = torch.zeros((n, n, n, 16), dtype=torch.float64, device=DEV)
    act[..., 0], act[..., 1] = delta, phi
    p = torch.as_tensor(params, dtype=torch.float64, device=DEV).view(3, 27 * 256 + 16)
    for l in range(3):
        w, bias = p[l, : 27 * 256].view(27, 16, 16), p[l, 27 * 256:]
        nxt = bias.expand(n, n, n, 16).clone()
        for t in range(27):
            off = (1 - t // 9, 1 - t // 3 % 3, 1 - t % 3)
            nxt += torch.roll(act, off, dims=(0, 1, 2)) @ w[t]
        act = nxt if l == 2 else torch.where(nxt > 0, nxt, 0.1 * nxt)
    o = act[..., :3].reshape(-1, 3)
    out = torch.zeros((len(x), 3), dtype=torch.float64, device=DEV)
    for cell, w in _corners(x, n, L):
        out += o[cell] * w[:, None]
    return out


def exact(case, seed):
    kind, nc, n = case["kind"], case["nc"], case["ngrid"]
    L = float(np.float32(case["boxsize"]))
    # the halo finder and the random field of the initial conditions have no
    # plain torch counterpart; a first optimiser step divides every gradient
    # by its own size, so its sign alone decides
    if kind in ("fof", "lpt", "train"):
        return None
    if kind == "batch":
        out = []
        for i, sp in enumerate(_batch_specs(case)):
            w = _particles(nc, sp["boxsize"], seed + 1009 * i, "ics")
            d, v, x = _realization_exact(w, nc, n, sp["boxsize"], 0.02, sp["nsteps"], True)
            out.append({"displacement": d, "v": v, "id": None,
                        "pk": _power_exact(x, nc, n, sp["boxsize"])[1]})
        return out
    if kind == "run":
        w = _particles(nc, L, seed, "ics")
        d, v, _ = _realization_exact(w, nc, n, L, 0.02, case["steps"], False)
        return {"displacement": d, "v": v, "id": None}
    w = _particles(nc, L, seed, case.get("stage", "late"))
    x = w.view(torch.float32)[:, 0:3].double()
    del w
    if kind == "pk":
        return list(_power_exact(x, nc, n, L))
    if kind == "force":
        return _force_exact(x, nc, n, L, case["gradient"], case["laplacian"], case["deconvolve"],
                            _knots(case["knots"], n, seed))
    f, delta = _force_exact(x, nc, n, L, delta=True)
    c = _net_exact(x, delta, _net_params(seed, 3 * (27 * 256 + 16)), n, L)
    return [f[a] + c[:, a] for a in range(3)]
