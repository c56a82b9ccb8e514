"""The run-time-plan passes (csrc/passes.cuh, csrc/long1d.cuh) at the edges of
their plans and tiles: one and two stages, primes with and without a stage
before them, primes above the size of the coefficient table, lines fewer than
a tile, the 1D split's extremes, rows that leave the tile for the in-place
kernel.  FP64 against the oracle (pocketfft) within 1e-12 relative; mixed
precision against the FP64 solve."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

SIZES = [
    # 1D: M = 1, 2, primes (Q = 1), a prime above the table, P = 4093 (one unpadded row), odd splits
    (2,), (4,), (6,), (26,), (62,), (134,), (254,), (4078,), (16372,), (4098,), (4096,), (4100,), (777600,), (2 * 641 * 769,),
    # 2D: radix 1, single stages, primes 11, 13, 31, 41, 67, 127, lines and rows fewer than a tile
    (2, 2), (4, 22), (22, 4), (26, 134), (310, 22), (62, 82), (254, 14), (14, 254), (462, 462), (720, 462), (1022, 6),
    (96, 1000), (1000, 96), (11000, 4), (16384, 4), (6, 2048),
    # 3D
    (62, 82, 26), (22, 14, 34), (2, 2, 2), (310, 82, 10), (48, 44, 52), (30, 98, 22),
]


def relerr(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


def model(size, keep, seed, **opts):
    import csipm
    import torch
    rng = np.random.default_rng(seed)
    N = int(np.prod(size))
    z0 = rng.standard_normal(N)
    lam = 0.1
    missing = None
    if keep is not None:
        z0 = np.where(keep, z0, 0.0)
        missing = np.flatnonzero(~keep)
    return csipm.FFTNLPModel(csipm.FFTParameters(len(size), size, torch.tensor(z0, device="cuda"), lam, missing), rdft=True,
                             **opts)


@pytest.mark.parametrize("size", SIZES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("autotune", [False, True])
def test_products(cuda, size, autotune):
    torch = cuda
    if autotune and len(size) == 1:
        pytest.skip("1D passes are not tuned")
    N = int(np.prod(size))
    rng = np.random.default_rng(N)
    for masked in (False, True):
        keep = (rng.random(N) > 0.2) if masked else None
        nlp = model(size, keep, 5, autotune=autotune)
        op, ref = nlp.op_fft, O.Operator(size, keep)
        x = rng.standard_normal(N)
        xt = torch.tensor(x, device="cuda")
        assert relerr(op.M_perp_beta(xt).cpu().numpy(), ref.A(x)) <= 1e-12
        assert relerr(op.M_perpt_z(xt).cpu().numpy(), ref.At(x)) <= 1e-12
        assert relerr(op.M_perpt_M_perp_vec(xt).cpu().numpy(), ref.AtA(x)) <= 1e-12
        op.close()


@pytest.mark.parametrize("kind,dims", [("1d", (4078,)), ("1d", (24010,)), ("2d", (62, 82)), ("2d", (134, 26)),
                                       ("2d", (96, 1000)), ("3d", (22, 14, 34)), ("3d", (48, 44, 52))])
@pytest.mark.parametrize("layout", ["solver", "reference"])
def test_solves(cuda, kind, dims, layout):
    """The FP64 and FP32 passes inside a solve, in both orders of the vectors,
    at the bounds of the mixed-precision tests (beta 1e-6, objective 1e-8)."""
    import csipm
    import csipm.problems as P
    torch = cuda
    spec = P.make_spec(kind, dims=dims, seed=5)
    op0 = O.Operator(spec.size)
    prob = P.finalize(spec, op0.A, op0.At)
    got = {}
    for precision in ("fp64", "mixed"):
        params = csipm.FFTParameters(len(dims), dims, torch.tensor(prob.z0, device="cuda"), prob.lam, prob.missing)
        nlp = csipm.FFTNLPModel(params, rdft=True, precision=precision, tol=1e-10, ipm_cg_rtol=1e-2, layout=layout)
        r = csipm.ipm_solve(nlp)
        assert r.status == 0, r.stats
        got[precision] = (r.beta.cpu().numpy(), r.stats["lasso_obj"])
        nlp.op_fft.close()
    assert relerr(got["mixed"][0], got["fp64"][0]) <= 1e-6
    assert abs(got["mixed"][1] - got["fp64"][1]) <= 1e-8 * abs(got["fp64"][1])
