"""Timed workloads of the library: what programs built on it ask of it, from the
smallest call to the largest.

Every case goes through the public entry points (itp2d_b200.capi.Context, one
device-resident state set, and itp2d_b200.system.ITPSystem, the native driver).
States and outputs stay on the device unless the entry point itself works on
host data. ``exact`` restates the same operators in plain 64-bit torch.

    propagate   one imaginary time step of every state (multi-product split)
    energies    expectation value and deviation of H for every state
    canonical   subspace orthonormalisation S = U l U^H, psi' = psi U l^{-1/2}
    cholesky    orthonormalisation in Gram-Schmidt order, psi' = psi L^{-H}
    step        propagate + canonical + energies: one iteration of a solve
    solve       a whole solve from noise with the native driver
"""
import math

import numpy as np
import torch

from itp2d_b200 import capi
from itp2d_b200.system import ITPSystem, Parameters

FP = {"fp64": capi.FP64, "fp32": capi.FP32}
CPLX = {"fp64": torch.complex128, "fp32": torch.complex64}


def _case(name, op, sx, sy, k, precision="fp64", boundary="periodic", B=0.0, m=2, eps=0.05, length=12.0, bumps=0,
          engine="dmma"):
    c = dict(op=op, sx=sx, sy=sy, k=k, precision=precision, boundary=boundary, B=B, m=m, eps=eps, length=length,
             bumps=bumps, engine=engine)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the driver's default problem (64 x 64, 25 states, 10th order): launch latency
        _case("propagate_64_k25_m5", "propagate", 64, 64, 25, m=5),
        # hard walls (sine transforms), second order: the harmonic box of 64 states
        _case("propagate_dirichlet_128_k64", "propagate", 128, 128, 64, boundary="dirichlet", m=1, eps=0.02),
        # one instance of a batch of uneven dots: lines that are no power of two, single precision
        _case("propagate_192x160_k77_fp32", "propagate", 192, 160, 77, "fp32", B=1.3, m=2, bumps=20),
        # the magnetic dot: 500 states in a field, 4th order
        _case("propagate_256_k500", "propagate", 256, 256, 500, B=1.0, m=2, length=14.0),
        # the bumpy dot's single-precision sweeps: 2000 states, 6th order
        _case("propagate_512_k2000_fp32", "propagate", 512, 512, 2000, "fp32", B=0.5, m=3, length=16.0, bumps=400),
        # the convergence check of a large field-free set
        _case("energies_512_k700", "energies", 512, 512, 700, length=16.0, bumps=100),
        # one iteration of a served request (128 x 128, 200 states)
        _case("step_128_k200", "step", 128, 128, 200, B=0.7, m=2, bumps=30),
        # the magnetic dot's orthonormalisation, FP64 tensor cores
        _case("canonical_256_k500", "canonical", 256, 256, 500, B=1.0, length=14.0),
        # the refinement's orthonormalisation on the int8 tensor cores
        _case("canonical_512_k1000_int8", "canonical", 512, 512, 1000, B=0.5, length=16.0, engine="int8"),
        # the bumpy dot's orthonormalisation between canonical steps
        _case("cholesky_512_k2000_fp32", "cholesky", 512, 512, 2000, "fp32", B=0.5, length=16.0),
        # a small solve to 1e-9, where host work and launches count
        _case("solve_96_k48", "solve", 96, 96, 48, B=0.8, m=2, bumps=10),
        # the magnetic dot in the mixed form: single-precision sweeps, FP64 refinement on int8 tensor cores
        _case("solve_256_k500_mixed", "solve", 256, 256, 500, "fp32", B=1.0, m=2, length=14.0, engine="int8"),
    ]


def draw(rng):
    op = rng.choice(["propagate", "propagate", "propagate", "energies", "step", "canonical", "cholesky", "solve"])
    precision = rng.choice(["fp64", "fp32"])
    sizes = [48, 64, 80, 96, 100, 108, 128, 128, 144, 160, 192, 200, 256, 256, 320, 384, 512, 512]
    sx = rng.choice(sizes)
    # most grids are square; a rectangle has the neighbouring sizes
    sy = sx if rng.random() < 0.7 else rng.choice([n for n in sizes if sx / 2 <= n <= 2 * sx])
    G = sx * sy
    top = min(2000, G // 16)
    k = int(round(math.exp(rng.uniform(math.log(16), math.log(top)))))
    if op in ("step", "canonical", "cholesky"):
        # k^2 G of the contractions up to that of 1000 states on 512 x 512
        k = min(k, int(math.sqrt(1000.0 ** 2 * 512 ** 2 / G)))
        if op == "step":
            precision = "fp64"
            k = min(k, 600)
    if op == "canonical":
        precision = "fp64"
    if op == "solve":
        sx = sy = rng.choice([64, 96, 128, 160, 192])
        k = rng.randint(16, 96)
        precision = "fp64"
    boundary = "dirichlet" if op == "propagate" and rng.random() < 0.2 and G <= 200 * 200 else "periodic"
    B = 0.0 if boundary == "dirichlet" or rng.random() < 0.35 else round(rng.uniform(0.2, 2.0), 3)
    m = 1 if boundary == "dirichlet" else rng.choice([1, 2, 2, 2, 3])
    if op == "solve":
        m = 2
    length = 16.0 if sx >= 384 else 14.0 if sx >= 200 else 12.0
    bumps = rng.choice([0, rng.randint(1, 50)])
    engine = "int8" if op == "canonical" and k >= 128 and rng.random() < 0.5 else "dmma"
    return _case(None, op, sx, sy, k, precision, boundary, B, m, 0.02 if m == 1 else 0.05, length, bumps, engine)


# ---- inputs ---------------------------------------------------------------------------------------------------

def _positions(c):
    dx = c["length"] / c["sx"]
    x = (2 * torch.arange(c["sx"], dtype=torch.float64, device="cuda") + 1 - c["sx"]) * (0.5 * dx)
    y = (2 * torch.arange(c["sy"], dtype=torch.float64, device="cuda") + 1 - c["sy"]) * (0.5 * dx)
    return dx, x, y


def _impurities(c, seed):
    """Rows (x, y, A, w): bumps within half the box, amplitude 0.8..1.2."""
    g = np.random.default_rng([seed, 7])
    n, half = c["bumps"], 0.375 * c["length"]
    w = np.full(n, 0.1) if n > 50 else g.uniform(0.1, 0.3, n)
    return np.column_stack([g.uniform(-half, half, (n, 2)), g.uniform(0.8, 1.2, n), w])


def _bumps(c, seed):
    _, x, y = _positions(c)
    V = torch.zeros(c["sy"], c["sx"], dtype=torch.float64, device="cuda")
    for bx, by, A, w in _impurities(c, seed).tolist():
        V += A * torch.exp(-((y - by) ** 2)[:, None] / (2 * w * w)) * torch.exp(-((x - bx) ** 2)[None, :] / (2 * w * w))
    return V


def _potential(c, seed):
    """Harmonic dot plus bumps. The energy zero is moved to about the lowest
    level, so that states which are propagated again and again without being
    normalised keep their size."""
    _, x, y = _positions(c)
    V = 0.5 * (x[None, :] ** 2 + y[:, None] ** 2) + _bumps(c, seed)
    return V - math.sqrt(1.0 + 0.25 * c["B"] ** 2) - 0.3 * min(1.0, c["bumps"] / 100)


def _states(c, seed):
    """Smooth random states, nearly orthogonal: noise with the upper half of
    the wavenumbers damped, state n weighted by exp(-eps E_n) like an
    orthonormal set after one time step."""
    dt, k, sy, sx = CPLX[c["precision"]], c["k"], c["sy"], c["sx"]
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    fy = torch.fft.fftfreq(sy, device="cuda", dtype=torch.float64)
    fx = torch.fft.fftfreq(sx, device="cuda", dtype=torch.float64)
    damp = torch.exp(-(fy[:, None] ** 2 + fx[None, :] ** 2) / 0.25 ** 2).to(dt)
    psi = torch.empty(k, sy, sx, dtype=dt, device="cuda")
    dx = c["length"] / sx
    for a in range(0, k, 128):
        b = min(k, a + 128)
        z = torch.randn(b - a, sy, sx, dtype=dt, device="cuda", generator=g)
        z = torch.fft.ifft2(z * damp)
        n = torch.arange(a, b, dtype=torch.float64, device="cuda")
        size = torch.exp(-c["eps"] * torch.sqrt(2 * n)) / dx
        z *= (size / torch.linalg.vector_norm(z, dim=(1, 2)).double()).to(dt)[:, None, None]
        psi[a:b] = z
    return psi


class _DeviceArray:
    """Device memory of a context; a tensor made of it keeps the context."""

    def __init__(self, ctx, ptr, shape, typestr):
        self.ctx = ctx
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 3}


def _view(state):
    """The context's state array as a tensor (the library swaps buffers)."""
    ptr = state["ctx"].device_states()
    t = state["views"].get(ptr)
    if t is None:
        c = state["case"]
        t = torch.as_tensor(_DeviceArray(state["ctx"], ptr, (c["k"], c["sy"], c["sx"]),
                                         "<c16" if c["precision"] == "fp64" else "<c8"), device="cuda")
        state["views"][ptr] = t
    return t


def prepare(case, seed):
    c = case
    if c["op"] == "solve":
        return _prepare_solve(c, seed)
    stream = torch.cuda.Stream()
    ctx = capi.Context(c["sx"], c["sy"], c["length"] / c["sx"], c["k"],
                       capi.DIRICHLET if c["boundary"] == "dirichlet" else capi.PERIODIC, c["B"], c["m"],
                       FP[c["precision"]], stream=stream.cuda_stream)
    ctx.set_potential(_potential(c, seed).cpu().numpy())
    ctx.set_time_step(c["eps"])
    if c["engine"] == "int8":
        ctx.set_fp64_engine(capi.FP64_INT8)
    state = {"case": c, "ctx": ctx, "stream": stream, "views": {}, "psi": _states(c, seed)}
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        _view(state).copy_(state["psi"])
    stream.synchronize()
    if c["op"] in ("propagate", "energies"):
        state["psi"] = None  # works on the resident states
    return state


def _prepare_solve(c, seed):
    k, sy, sx = c["k"], c["sy"], c["sx"]
    mixed = c["precision"] == "fp32"
    p = Parameters(sx=sx, sy=sy, length=c["length"], boundary=capi.PERIODIC, B=c["B"], halforder=c["m"], num_states=k,
                   wanted=k // 2, eps=[c["eps"]], exhaust_eps=False, max_steps=200, potential="harmonic",
                   timestep_test="abschange(1e-9)", final_test="abschange(1e-9)")
    if mixed:
        p.precision, p.fp32_switch, p.fp32_canonical_every = capi.FP32, 1e-7, 3
        p.fp32_between, p.fp32_switch_span, p.fp64_engine = capi.BETWEEN_CHOLESKY, 3, capi.FP64_INT8
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    psi = torch.randn(k, sy, sx, dtype=torch.complex128, device="cuda", generator=g)
    host = torch.empty(k, sy, sx, dtype=torch.complex128, pin_memory=True)
    host.copy_(psi)
    system = ITPSystem(p, extra_potential=_bumps(c, seed).cpu().numpy(), init_states=host.numpy())
    return {"case": c, "system": system, "init": host, "wanted": k // 2}


def run(state):
    c, op = state["case"], state["case"]["op"]
    if op == "solve":
        # the driver takes host states: a new start, then to convergence
        system = state["system"]
        system.reset(state["init"].numpy())
        system.run()
        return {"E": system.energies()[0][:state["wanted"]]}
    ctx = state["ctx"]
    if op == "propagate":
        ctx.propagate()
        return {"psi": _view(state)}
    if op == "energies":
        E, sigma, _, _ = ctx.energies()
        return _spectrum(c, E, sigma)
    with torch.cuda.stream(state["stream"]):
        _view(state).copy_(state["psi"])
        if op == "cholesky":
            ctx.orthonormalize(capi.ORTHO_CHOLESKY)
            return {"psi": _view(state)}
        out = {}
        if op == "step":
            ctx.propagate()
        ctx.orthonormalize()
        if op == "step":
            E, sigma, _, _ = ctx.energies()
            out = _spectrum(c, E, sigma)
        # the phase of an eigenvector is arbitrary: what a program reads is the modulus
        out["modulus"] = _view(state).abs()
        return out


def _spectrum(c, E, sigma):
    # single-precision states give energies of that precision
    t = np.float64 if c["precision"] == "fp64" else np.float32
    return {"E": E.astype(t), "sigma": sigma.astype(t)}


# ---- work and 64-bit results --------------------------------------------------------------------------------------

def work(case):
    c = case
    b = 16 if c["precision"] == "fp64" else 8
    k, G = c["k"], c["sx"] * c["sy"]
    # forward and inverse transform along both axes, and the factor in between
    fft2 = k * G * (10.0 * (math.log2(c["sx"]) + math.log2(c["sy"])) + 4)
    prop = c["m"] * (c["m"] + 1) / 2 * fft2 + 6.0 * c["m"] * k * G
    energy = fft2 + 24.0 * k * G
    chol = 8.0 * k * k * G + 4.0 * k ** 3
    canon = 12.0 * k * k * G + 40.0 * k ** 3
    if c["op"] == "propagate":
        return {"bytes": 2.0 * k * G * b, "flops": prop}
    if c["op"] == "energies":
        return {"bytes": 1.0 * k * G * b, "flops": energy}
    if c["op"] == "cholesky":
        return {"bytes": 2.0 * k * G * b, "flops": chol}
    if c["op"] == "canonical":
        return {"bytes": (2.0 * b + b / 2) * k * G, "flops": canon}
    if c["op"] == "step":
        return {"bytes": (2.0 * b + b / 2) * k * G, "flops": prop + canon + energy}
    # a solve from noise takes ten iterations at the least
    return {"bytes": 16.0 * k * G, "flops": 10 * (prop + canon + energy)}


def _sine(n):
    """DST-II and its inverse (DST-III / 2n) as matrices."""
    j = torch.arange(n, dtype=torch.float64, device="cuda")
    D = 2 * torch.sin(math.pi * (j[:, None] + 1) * (2 * j[None, :] + 1) / (2 * n))
    inv = D.T / (2.0 * n)
    inv[:, -1] *= 0.5
    return D.to(torch.complex128), inv.to(torch.complex128)


def _wavenumbers(c):
    def axis(n, size):
        j = torch.arange(n, dtype=torch.float64, device="cuda")
        if c["boundary"] == "dirichlet":
            return (j + 1) * math.pi / size
        return torch.where(j < n // 2, j, j - n) * 2 * math.pi / size
    dx = c["length"] / c["sx"]
    return axis(c["sx"], c["length"]), axis(c["sy"], c["sy"] * dx)


def _exp_kinetic(c, e):
    """exp(-e T) on a chunk of states, T in the linear gauge A = (-B y, 0, 0)."""
    kx, ky = _wavenumbers(c)
    if c["B"] == 0:
        mult = torch.exp(-0.5 * e * (kx[None, :] ** 2 + ky[:, None] ** 2))
        if c["boundary"] == "dirichlet":
            (Dx, Ix), (Dy, Iy) = _sine(c["sx"]), _sine(c["sy"])
            return lambda a: Iy @ ((Dy @ a @ Dx.T) * mult) @ Ix.T
        return lambda a: torch.fft.ifft2(torch.fft.fft2(a) * mult)
    _, _, y = _positions(c)
    z = c["B"] * e
    X = torch.exp(-0.5 * e * math.tanh(z / 2) / z * (kx[None, :] - c["B"] * y[:, None]) ** 2)
    Y = torch.exp(-0.5 * e * math.sinh(z) / z * ky ** 2)[:, None]

    def apply(a):
        a = torch.fft.fft(a, dim=-1) * X
        a = torch.fft.ifft(torch.fft.fft(a, dim=-2) * Y, dim=-2)
        return torch.fft.ifft(a * X, dim=-1)
    return apply


def _chunks(c):
    step = max(1, (1 << 26) // (c["sx"] * c["sy"]))
    return [slice(a, min(c["k"], a + step)) for a in range(0, c["k"], step)]


def _propagated(c, V, psi):
    """sum_t c_t [exp(-e_t V/2) exp(-e_t T) exp(-e_t V/2)]^t, e_t = eps / t."""
    members = []
    for t in range(1, c["m"] + 1):
        e = c["eps"] / t
        coef = float(t) ** (2 * (c["m"] - 1))
        for n in range(1, c["m"] + 1):
            coef /= t * t - n * n if n != t else 1
        members.append((t, coef, torch.exp(-0.5 * e * V), _exp_kinetic(c, e)))
    out = torch.empty(psi.shape, dtype=torch.complex128, device="cuda")
    for s in _chunks(c):
        a = psi[s].to(torch.complex128)
        total = torch.zeros_like(a)
        for t, coef, half, kin in members:
            b = a
            for _ in range(t):
                b = half * kin(half * b)
            total += coef * b
        out[s] = total
    return out


def _energies(c, V, psi):
    kx, ky = _wavenumbers(c)
    dx, _, y = _positions(c)
    E, sigma = [], []
    for s in _chunks(c):
        a = psi[s].to(torch.complex128)
        if c["B"] == 0:
            h = torch.fft.ifft2(torch.fft.fft2(a) * (0.5 * (kx[None, :] ** 2 + ky[:, None] ** 2)))
        else:
            h = torch.fft.ifft(torch.fft.fft(a, dim=-1) * (0.5 * (kx[None, :] - c["B"] * y[:, None]) ** 2), dim=-1)
            h += torch.fft.ifft(torch.fft.fft(a, dim=-2) * (0.5 * ky ** 2)[:, None], dim=-2)
        h += V * a
        mean = (a.conj() * h).sum((1, 2)).real * dx * dx
        sq = (h.abs() ** 2).sum((1, 2)) * dx * dx
        if c["precision"] == "fp32":  # Rayleigh quotients
            n = (a.abs() ** 2).sum((1, 2)) * dx * dx
            mean, sq = mean / n, sq / n
        E.append(mean)
        sigma.append(torch.sqrt(torch.clamp(sq - mean * mean, min=0)))
    return {"E": torch.cat(E).cpu().numpy(), "sigma": torch.cat(sigma).cpu().numpy()}


def _combined(c, psi, W):
    flat = psi.reshape(c["k"], -1)
    out = torch.empty(c["k"], flat.shape[1], dtype=torch.complex128, device="cuda")
    for a in range(0, flat.shape[1], 1 << 15):
        b = min(flat.shape[1], a + (1 << 15))
        out[:, a:b] = W.T @ flat[:, a:b].to(torch.complex128)
    return out.reshape(psi.shape)


def exact(case, seed):
    c = case
    if c["op"] == "solve":
        return None
    V, psi = _potential(c, seed), _states(c, seed)
    if c["op"] == "propagate":
        return {"psi": _propagated(c, V, psi)}
    if c["op"] == "energies":
        return _energies(c, V, psi)
    if c["op"] == "step":
        psi = _propagated(c, V, psi)
    dx = c["length"] / c["sx"]
    flat = psi.reshape(c["k"], -1)
    S = torch.zeros(c["k"], c["k"], dtype=torch.complex128, device="cuda")
    for a in range(0, flat.shape[1], 1 << 15):
        f = flat[:, a:a + (1 << 15)].to(torch.complex128)
        S += f.conj() @ f.T
    S *= dx * dx
    if c["op"] == "cholesky":
        L = torch.linalg.cholesky(S)
        eye = torch.eye(c["k"], dtype=torch.complex128, device="cuda")
        return {"psi": _combined(c, psi, torch.linalg.solve_triangular(L, eye, upper=False).conj().T.contiguous())}
    lam, U = torch.linalg.eigh(S)
    psi = _combined(c, psi, U / torch.sqrt(lam))
    out = _energies(c, V, psi) if c["op"] == "step" else {}
    out["modulus"] = psi.abs()
    return out
