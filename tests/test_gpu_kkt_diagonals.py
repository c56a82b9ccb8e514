"""solve_kkt! on diagonals the N-unknown form does not serve: the 2N method's
iterates on the K that build_kkt! stored, with and without the preconditioner
and in both orders of the vectors, against the numpy statement of that method.

Bound: as for the N-unknown iterates (test_gpu_newton.py), 1e-9 relative."""
import numpy as np
import pytest

import oracle as O
import oracle_ipm as OI

pytestmark = pytest.mark.gpu


def _system(torch, size, **opts):
    import csipm
    N = int(np.prod(size))
    rng = np.random.default_rng(N)
    keep = rng.random(N) > 0.2
    z0 = np.where(keep, rng.standard_normal(N), 0.0)
    params = csipm.FFTParameters(len(size), size, torch.tensor(z0, device="cuda"), 0.3, np.flatnonzero(~keep))
    nlp = csipm.FFTNLPModel(params, rdft=True, cg_atol=0.0, **opts)
    return nlp, csipm.FFTKKTSystem(nlp), O.Operator(size, keep), rng


def _close(got, want):
    return np.linalg.norm(got - want) <= 1e-9 * np.linalg.norm(want)


@pytest.mark.parametrize("size", [(200,), (62, 82), (22, 14, 34)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("pc", [True, False])
@pytest.mark.parametrize("layout", ["solver", "reference"])
@pytest.mark.parametrize("entries", ["all", "one"])
def test_diagonals_other_than_the_built_ones(cuda, size, pc, layout, entries):
    """solve_kkt!(w, pr_diag) with another pr_diag than build_kkt!: K and P stay
    the built ones, the right-hand side and the back-substitution take pr_diag."""
    torch = cuda
    nlp, kkt, op, rng = _system(torch, size, cg_rtol=1e-2, preconditioner=pc, layout=layout)
    N = op.N
    built = np.ones(4 * N)
    built[2 * N:] = 10.0 ** rng.uniform(-1.0, 1.0, 2 * N)
    pr = built.copy()
    if entries == "all":
        pr[2 * N:] *= 1.0 + rng.random(2 * N)
    else:
        pr[2 * N + N // 3] *= 2.0
    kkt.build_kkt(torch.tensor(built, device="cuda"))
    w = rng.standard_normal(6 * N)
    wt = torch.tensor(w, device="cuda")
    kkt.solve_kkt(wt, torch.tensor(pr, device="cuda"))
    sol, it = OI.kkt_solve(op, OI.kkt_build(built, N), w, pr, atol=0.0, rtol=1e-2, preconditioner=pc)
    assert kkt.krylov_iterations[-1] == it
    assert _close(wt.cpu().numpy(), sol)
    nlp.op_fft.close()


def _cg_2n(op, K, b, steps):
    """`steps` iterations of the preconditioned CG on 2N unknowns, whatever the
    signs of p.q and r.z."""
    n2 = b.size
    mul = lambda v: OI.condensed_mul(op, K, np.zeros(n2), v, 1.0, 0.0)
    pre = lambda v: OI.precond_mul(K, np.zeros(n2), v, 1.0, 0.0)
    x, r = np.zeros(n2), b.copy()
    p = pre(r)
    rz = r @ p
    for _ in range(steps):
        q = mul(p)
        a = rz / (p @ q)
        x += a * p
        r -= a * q
        z = pre(r)
        rz, old = r @ z, rz
        p = z + rz / old * p
    return x


@pytest.mark.parametrize("size", [(200,), (62, 82), (22, 14, 34)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("layout", ["solver", "reference"])
@pytest.mark.parametrize("diag", ["negative", "opposite", "zero"])
def test_diagonals_that_are_not_positive(cuda, size, layout, diag):
    """K is indefinite (negative), a pair of diagonals sums to zero (opposite),
    or one of each pair is zero: three iterations and no error, as the 2N method."""
    torch = cuda
    nlp, kkt, op, rng = _system(torch, size, cg_rtol=0.0, cg_maxit=3, layout=layout)
    N = op.N
    S1, S2 = 1.0 + rng.random(N), 1.0 + rng.random(N)
    if diag == "negative":
        S1, S2 = -2.0 - S1, -2.0 - S2
    elif diag == "opposite":
        S2[::7] = -S1[::7]
    else:
        S2[::3] = 0.0
    pr = np.concatenate([np.ones(2 * N), S1, S2])
    prt = torch.tensor(pr, device="cuda")
    kkt.build_kkt(prt)
    # w3, w5 and w6 zero: b = [w1 + w4; w2 - w4], and no 0/0 in the back-substitution
    w = rng.standard_normal((6, N))
    w[2] = w[4] = w[5] = 0.0
    wt = torch.tensor(w.reshape(-1), device="cuda")
    kkt.solve_kkt(wt, prt)
    assert kkt.krylov_iterations == [3]
    x = _cg_2n(op, OI.kkt_build(pr, N), np.concatenate([w[0] + w[3], w[1] - w[3]]), 3)
    got = wt.cpu().numpy()
    assert _close(got[:2 * N], x)
    nlp.op_fft.close()
