"""The work a user of this package has it do, as timed cases.

Every case goes through the public entry points of ``csipm`` (the Python mirror
of the C ABI): products with the masked operator, evaluations of the NLP model,
the KKT plugin's condensed product and Newton solve, whole interior-point
recoveries, and a batch of recoveries.  Sizes are those of the measured
workloads (1D 2^14, 2D 1024^2, 3D 256^3 and 320^3), of the serving stream (1D
from 2^12 to 2^20, 2D sides from 128 to 1024, 3D sides from 32 to 128), and the
grid of the largest volume the method is used on (310 x 410 x 410, whose sides
have the prime factors 31 and 41).

Signals have a sparse half spectrum plus noise; the missing samples are gaps
(1D), disks on a lattice plus random pixels (2D) or balls on a lattice (3D).
"""
import itertools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "compressedsensingipm.jl_b200"))
import csipm  # noqa: E402

DEV = "cuda" if torch.cuda.is_available() else "cpu"

# share of nonzero spectrum entries, lambda / |A'z0|_inf, by dimension
SPARSITY = {1: 0.02, 2: 0.01, 3: 0.005}
LAM = {1: 0.1, 2: 0.1, 3: 0.05}


def _case(name, do, n1, n2=1, n3=1, **more):
    return {"name": name, "do": do, "n1": n1, "n2": n2, "n3": n3, **more}


def listed():
    return [
        # the smallest call: one A'A product on the shortest rows of the serving range (launch latency)
        _case("product 1D 4096", "product", 4096),
        # a long ragged row, 2^7 * 3^5 * 5^2 samples: the transform does not fit one block
        _case("product 1D 777600", "product", 777600),
        # synthesis and analysis of an image, A then A', as a driver makes and inspects its data
        _case("A and A' 2D 1024x1024", "synthesis", 1024, 1024),
        # the product on the grid of the largest real volume (sides with the factors 31 and 41)
        _case("product 3D 310x410x410", "product", 310, 410, 410),
        # obj, grad and cons of one iterate, as a line search asks for them, on a ragged image
        _case("model 2D 720x462", "model", 720, 462),
        # the KKT plugin: condensed K x with alpha and beta on the 256^3 crystal grid
        _case("condensed 3D 256", "condensed", 256, 256, 256),
        # the KKT plugin: one Newton system, built and solved to the reference's tolerance
        _case("Newton solve 3D 128x120x96", "newton", 128, 120, 96),
        # whole recoveries at the measured workloads
        _case("recovery 1D 16384", "recovery", 16384, precision="fp64", tol=1e-8, rtol=1e-2),
        _case("recovery 2D 1024x1024", "recovery", 1024, 1024, precision="fp64", tol=1e-8, rtol=1e-2),
        _case("recovery 3D 256 fp64", "recovery", 256, 256, 256, precision="fp64", tol=1e-8, rtol=1e-2),
        _case("recovery 3D 320 mixed", "recovery", 320, 320, 320, precision="mixed", tol=1e-10, rtol=1e-2),
        # a server's batch: recoveries of small images of uneven sizes, solved together
        _case("batch 16 x 2D 128-256", "batch", 128, 256, count=16, tol=1e-8, rtol=1e-3),
    ]


def _even(rng, lo, hi, primes):
    """A log-uniform draw from [lo, hi] moved to the nearest even number with these prime factors."""
    x = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    found = [v for v in _even_numbers(lo, hi, primes)]
    return min(found, key=lambda v: abs(math.log(v / x)))


def _even_numbers(lo, hi, primes):
    got, front = set(), {2}
    while front:
        front = {v * p for v in front for p in primes if v * p <= hi} - got
        got |= front
    return sorted(v for v in got | {2} if lo <= v <= hi)


def draw(rng):
    do = rng.choice(["product", "product", "synthesis", "model", "condensed", "newton", "recovery", "recovery", "batch"])
    if do == "batch":
        lo = _even(rng, 128, 180, (2, 3, 5))
        return {"do": do, "n1": lo, "n2": _even(rng, lo + 40, 256, (2, 3, 5)), "n3": 1, "count": rng.randint(8, 16),
                "tol": 1e-8, "rtol": 1e-3}
    dim = rng.choice([1, 2, 3])
    # products and evaluations also meet the sides of raw volumes: one more factor of 7, 11 or 31
    more = () if do in ("recovery", "newton") else ((7,), (7,), (11,), (31,))[rng.randrange(4)]
    if dim == 1:
        size = [_even(rng, 4096, 1 << 20, (2, 3, 5))]
    elif dim == 2:
        size = [_even(rng, 128, 1024, (2, 3, 5) + more) for _ in range(2)]
    else:
        hi = 128 if do in ("recovery", "newton") else 256
        size = [_even(rng, 32, hi, (2, 3, 5) + more) for _ in range(3)]
    size += [1] * (3 - dim)
    case = {"do": do, "n1": size[0], "n2": size[1], "n3": size[2]}
    if do == "recovery":
        case |= {"precision": rng.choice(["fp64", "mixed"]), "tol": 1e-8, "rtol": rng.choice([1e-2, 1e-3])}
    return case


# ------------------------------------------------------------------ inputs
def _size(case):
    s = (case["n1"], case["n2"], case["n3"])
    return s[:1] if s[1] == 1 else (s[:2] if s[2] == 1 else s)


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _rand(gen, *shape):
    return torch.rand(*shape, generator=gen, device=DEV, dtype=torch.float64)


def _randn(gen, *shape):
    return torch.randn(*shape, generator=gen, device=DEV, dtype=torch.float64)


def _keep(size, gen):
    """Observed samples, as an array of the grid's shape with dimension 1 last (fastest)."""
    shape = tuple(reversed(size))
    if len(size) == 1:   # 20 gaps that remove about 15%
        n = size[0]
        start = (_rand(gen, 20) * n).long().cpu().numpy()
        length = (_rand(gen, 20) * 2 * 0.0085 * n).long().cpu().numpy()
        keep = np.ones(n, dtype=bool)
        for a, m in zip(start, length):
            keep[a:a + m + 1] = False
        return torch.from_numpy(keep).to(DEV)
    period, radius = (32, 4) if len(size) == 2 else (16, 3)
    d2 = torch.zeros(shape, device=DEV, dtype=torch.int32)
    for axis, n in enumerate(shape):
        r = (torch.arange(n, device=DEV, dtype=torch.int32) - period // 2) % period
        r = torch.minimum(r, period - r) ** 2
        d2 += r.view([-1 if a == axis else 1 for a in range(len(shape))])
    keep = d2 > radius * radius
    if len(size) == 2:
        keep &= _rand(gen, *shape) >= 0.05
    return keep


def _signal(size, gen):
    """A real signal with a sparse half spectrum (N(0,1); log-normal with random signs in 3D) and noise 0.01."""
    dim, shape = len(size), tuple(reversed(size))
    half = shape[:-1] + (shape[-1] // 2 + 1,)
    x = torch.zeros(half, device=DEV, dtype=torch.complex128)
    k = max(1, int(2 * SPARSITY[dim] * x.numel()))
    # one place in each of k equal stretches: no place twice
    at = ((torch.arange(k, device=DEV) + _rand(gen, k)) * (x.numel() / k)).long().clamp_(max=x.numel() - 1)
    v = _randn(gen, k, 2)
    if dim == 3:
        v = torch.exp(v) * torch.sign(_rand(gen, k, 2) - 0.5)
    v = v * (_rand(gen, k, 2) < 0.5) * math.sqrt(0.5)
    x.view(-1)[at] = torch.complex(v[:, 0], v[:, 1])
    return torch.fft.irfftn(x, s=shape, norm="ortho") + 0.01 * _randn(gen, *shape)


def _problem(size, seed):
    """(z0, lambda, host indices of the missing samples, keep) of one recovery."""
    gen = _gen(seed)
    keep = _keep(size, gen)
    z0 = torch.where(keep, _signal(size, gen), 0.0)
    spec = torch.view_as_real(torch.fft.rfftn(z0, norm="ortho"))
    lam = LAM[len(size)] * math.sqrt(2.0) * float(spec.abs().max())
    missing = torch.nonzero(~keep.reshape(-1)).reshape(-1).cpu().numpy().astype(np.int64)
    return z0.reshape(-1), lam, missing, keep


def _model(size, seed, **opts):
    z0, lam, missing, _ = _problem(size, seed)
    params = csipm.FFTParameters(len(size), size, z0, lam, missing)
    return csipm.FFTNLPModel(params, rdft=True, **opts)


def _sides(case):
    """The uneven images of a batch: sides walk through the smooth even numbers of [n1, n2]."""
    s = _even_numbers(case["n1"], case["n2"], (2, 3, 5))
    return [(s[(3 * k) % len(s)], s[(5 * k + 1) % len(s)]) for k in range(case["count"])]


def _vectors(case, seed):
    """The vectors a call takes beside its handle, as a dict of tensors."""
    n = math.prod(_size(case))
    gen = _gen(seed + 7919)
    do = case["do"]
    if do in ("product", "synthesis"):
        return {"x": _randn(gen, n)}
    if do == "model":
        return {"x": torch.cat([_randn(gen, n), 1.0 + _rand(gen, n)])}
    if do in ("condensed", "newton"):
        # slack block of pr_diag: z/s of an iterate half way, six decades
        diag = torch.cat([torch.zeros(2 * n, device=DEV, dtype=torch.float64), 10.0 ** (6.0 * _rand(gen, 2 * n) - 3.0)])
        if do == "condensed":
            return {"diag": diag, "x": _randn(gen, 2 * n), "y": _randn(gen, 2 * n)}
        return {"diag": diag, "w": _randn(gen, 6 * n)}
    return {}


def prepare(case, seed):
    do = case["do"]
    if do == "batch":
        return {"do": do, "models": [_model(s, 100 * seed + k, tol=case["tol"], ipm_cg_rtol=case["rtol"])
                                     for k, s in enumerate(_sides(case))]}
    size = _size(case)
    if do == "recovery":
        return {"do": do, "model": _model(size, seed, precision=case["precision"], tol=case["tol"],
                                          ipm_cg_rtol=case["rtol"])}
    s = {"do": do, "model": _model(size, seed), **_vectors(case, seed)}
    if do in ("condensed", "newton"):
        s["kkt"] = csipm.FFTKKTSystem(s["model"])
        s["kkt"].build_kkt(s["diag"])
        s["out"] = torch.empty_like(s["x"] if do == "condensed" else s["w"])
    elif do == "model":
        s["g"], s["c"] = torch.empty_like(s["x"]), torch.empty_like(s["x"])
    return s


def run(state):
    do = state["do"]
    if do == "recovery":   # what is recovered: the coefficients
        return csipm.ipm_solve(state["model"]).beta
    if do == "batch":
        return [r.beta for r in csipm.ipm_solve_batch(state["models"])]
    m = state["model"]
    if do == "product":
        return csipm.M_perpt_M_perp_vec(m.op_fft, state["x"])
    if do == "synthesis":
        z = csipm.M_perp_beta(m.op_fft, state["x"])
        return z, csipm.M_perpt_z(m.op_fft, z)
    if do == "model":
        return m.obj(state["x"]), m.grad(state["x"], state["g"]), m.cons(state["x"], state["c"])
    if do == "condensed":
        y = state["out"].copy_(state["y"])
        return state["kkt"].condensed_mul(y, state["x"], alpha=1.0, beta=-0.5)
    # a Newton system: MadNLP rewrites w and the diagonal before each solve
    w = state["out"].copy_(state["w"])
    state["kkt"].build_kkt(state["diag"])
    return state["kkt"].solve_kkt(w, state["diag"])


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    if case["do"] == "batch":
        each = [work({"do": "recovery", "n1": a, "n2": b, "n3": 1}) for a, b in _sides(case)]
        return {"bytes": sum(w["bytes"] for w in each), "flops": sum(w["flops"] for w in each)}
    n = math.prod(_size(case))
    fft = 2.5 * n * math.log2(n)              # one real transform
    mask = n / 8.0
    do = case["do"]
    if do == "product":                       # x in, y out
        return {"bytes": 16.0 * n + mask, "flops": 2 * fft}
    if do == "synthesis":                     # x in, z out and in, beta out
        return {"bytes": 32.0 * n + mask, "flops": 2 * fft}
    if do == "model":                         # beta, c and A'z0 in; g and constraints (2N each) out
        return {"bytes": 56.0 * n + mask, "flops": 2 * fft + 10.0 * n}
    if do == "condensed":                     # x, y, L1, L2 in, y out (and the copy into y)
        return {"bytes": 96.0 * n + mask, "flops": 2 * fft + 12.0 * n}
    if do == "newton":                        # w, diagonal in, w out; about 25 CG iterations on 2N vectors
        return {"bytes": 128.0 * n + mask, "flops": 25 * (2 * fft + 40.0 * n)}
    # a recovery: A'z0 in, beta out; about 10 iterations, 50 products
    return {"bytes": 16.0 * n + mask, "flops": 50 * (2 * fft) + 10 * 200.0 * n}


# ------------------------------------------------------------------ 64-bit answers
def _regions(dim):
    """The blocks of the coefficient vector in packing order, as one selector
    per dimension: 0 and 1 the self-conjugate positions 0 and N/2, "L" and "U"
    the positions below and above N/2.  Blocks without "L" hold real values,
    the others real parts, then imaginary parts, scaled by sqrt(2)."""
    b = (0, 1)
    if dim == 1:
        return [(0,), (1,), ("L",)]
    if dim == 2:
        return ([(i, j) for i in b for j in b] + [(i, "L") for i in b] + [("L", j) for j in b]
                + [("L", "L"), ("L", "U")])
    return ([(i, j, k) for i, j, k in itertools.product(b, b, b)]
            + [(i, j, "L") for i in b for j in b] + [(i, "L", k) for i in b for k in b]
            + [("L", j, k) for j in b for k in b]
            + [(i, s, "L") for i in b for s in "LU"] + [(s, j, "L") for j in b for s in "LU"]
            + [(s, "L", k) for k in b for s in "LU"]
            + [("L", "L", "L"), ("U", "L", "L"), ("L", "U", "L"), ("U", "U", "L")])


def _positions(size):
    """[(linear positions in the full spectrum, whether real)] of every block."""
    place = torch.arange(math.prod(size), device=DEV).view(tuple(reversed(size)))
    for reg in _regions(len(size)):
        cut = []
        for s, n in zip(reg, size):
            h = n // 2
            cut.append({0: slice(0, 1), 1: slice(h, h + 1), "L": slice(1, h), "U": slice(h + 1, n)}[s])
        yield place[tuple(reversed(cut))].reshape(-1), "L" not in reg


def _to_spectrum(beta, size):
    n, at = beta.numel(), 0
    x = torch.zeros(n, device=DEV, dtype=torch.complex128)
    mirror = torch.arange(n, device=DEV).view(tuple(reversed(size)))
    for axis in range(len(size)):
        mirror = torch.roll(torch.flip(mirror, (axis,)), 1, axis)
    mirror = mirror.reshape(-1)
    for pos, real in _positions(size):
        m = pos.numel()
        if real:
            x[pos] = beta[at:at + m].to(torch.complex128)
            at += m
        else:
            v = torch.complex(beta[at:at + m], beta[at + m:at + 2 * m]) * math.sqrt(0.5)
            x[pos] = v
            x[mirror[pos]] = v.conj()
            at += 2 * m
    return x.view(tuple(reversed(size)))


def _from_spectrum(x, size):
    x, got = x.reshape(-1), []
    for pos, real in _positions(size):
        v = x[pos]
        got += [v.real] if real else [math.sqrt(2.0) * v.real, math.sqrt(2.0) * v.imag]
    return torch.cat(got)


def _A(beta, size, keep):
    return torch.where(keep, torch.fft.ifftn(_to_spectrum(beta, size), norm="ortho").real, 0.0)


def _At(z, size):
    return _from_spectrum(torch.fft.fftn(z, norm="ortho"), size)


def exact(case, seed):
    do = case["do"]
    if do in ("recovery", "batch"):
        return None   # an iterate that meets the stopping test: no single value belongs to it
    size = _size(case)
    z0, lam, _, keep = _problem(size, seed)
    v = _vectors(case, seed)
    n = math.prod(size)

    def ata(b):
        return _At(_A(b, size, keep), size)

    if do == "product":
        return ata(v["x"])
    if do == "synthesis":
        z = _A(v["x"], size, keep)
        return z.reshape(-1), _At(z, size)
    if do == "model":
        be, c = v["x"][:n], v["x"][n:]
        q, b = ata(be), _At(z0.view(tuple(reversed(size))), size)
        return (float(0.5 * (be @ q) - be @ b + lam * c.sum()),
                torch.cat([q - b, torch.full_like(c, lam)]), torch.cat([-be - c, be - c]))
    s1, s2 = v["diag"][2 * n:3 * n], v["diag"][3 * n:]
    l1, l2 = s1 + s2, s1 - s2

    def condensed(x):
        return torch.cat([ata(x[:n]) + l1 * x[:n] + l2 * x[n:], l2 * x[:n] + l1 * x[n:]])

    if do == "condensed":
        return condensed(v["x"]) - 0.5 * v["y"]
    w1, w2, w3, w4, w5, w6 = v["w"].view(6, n)
    rhs = torch.cat([w1 - w3 + w4 - s1 * w5 + s2 * w6, w2 - w3 - w4 - s1 * w5 - s2 * w6])
    # eliminate the second half, then conjugate gradients with 1/(1 + D) until nothing moves
    d = l1 - l2 * l2 / l1
    f = rhs[:n] - l2 / l1 * rhs[n:]
    x, r = torch.zeros_like(f), f.clone()
    z = r / (1 + d)
    p, rz = z.clone(), r @ z
    stop = 1e-30 * float(rz)
    for _ in range(500):
        q = ata(p) + d * p
        a = rz / (p @ q)
        x += a * p
        r -= a * q
        z = r / (1 + d)
        rz, old = r @ z, rz
        if float(rz) <= stop:
            break
        p = z + rz / old * p
    y = (rhs[n:] - l2 * x) / l1
    w5 = -(w3 + s1 * (x + y + w5))
    w6 = -(w4 + s2 * (-x + y + w6))
    return torch.cat([x, y, (w3 + w5) / s1, (w4 + w6) / s2, w5, w6])
