"""1D products of the KKT plugins on both sides of the size from which their
epilogues take a pass of their own (l1d_last, csrc/long1d.cuh): half lengths odd
and even, lines of one and of several stages, against the oracle within 1e-12;
solves stopped after four CG iterations on 2N vectors within 1e-11."""
import numpy as np
import pytest

import oracle as O
import oracle_gondzio as OG
import oracle_ipm as OI

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


# 2^15 is the first with the pass of its own; 32766 = 2 3 43 127, 32770 = 2 5 29 113
@pytest.mark.parametrize("N", [32766, 32768, 32770, 45000, 65534, 777600])
def test_plugin_products(cuda, N):
    import csipm
    torch = cuda
    rng = np.random.default_rng(N)
    keep = rng.random(N) > 0.2
    z0 = np.where(keep, rng.standard_normal(N), 0.0)
    params = csipm.FFTParameters(1, (N,), torch.tensor(z0, device="cuda"), 0.3, np.flatnonzero(~keep))
    op = O.Operator((N,), keep)
    dev = lambda v: torch.tensor(v, device="cuda")
    opts = dict(rdft=True, cg_maxit=4, cg_atol=0.0)

    nlp = csipm.FFTNLPModel(params, preconditioner=False, **opts)
    kkt = csipm.FFTKKTSystem(nlp)
    pr = np.ones(4 * N)
    pr[2 * N:] = rng.uniform(0.05, 20.0, 2 * N)
    kkt.build_kkt(dev(pr))
    K = OI.kkt_build(pr, N)
    x, y = rng.standard_normal(6 * N), rng.standard_normal(6 * N)
    got = kkt.condensed_mul(dev(y[:2 * N]), dev(x[:2 * N]), 0.7, -0.4).cpu().numpy()
    assert rel(got, OI.condensed_mul(op, K, y[:2 * N], x[:2 * N], 0.7, -0.4)) <= 1e-12
    assert rel(kkt.mul(dev(y), dev(x), 0.7, -0.4).cpu().numpy(), OI.kkt_mul(op, y, x, 0.7, -0.4)) <= 1e-12
    sol, _ = OI.kkt_solve(op, K, x, pr, atol=0.0, rtol=0.0, preconditioner=False, itmax=4)
    assert rel(kkt.solve_kkt(dev(x), dev(pr)).cpu().numpy(), sol) <= 1e-11
    nlp.op_fft.close()

    gz = csipm.GondzioNLPModel(params, **opts)
    gk = csipm.GondzioKKTSystem(gz)
    gpr = rng.uniform(0.05, 4.0, 3 * N)
    gk.build_kkt(dev(gpr))
    G = OG.build(gpr, N)
    got = gk.condensed_mul(dev(y[:2 * N]), dev(x[:2 * N]), 0.7, -0.4).cpu().numpy()
    assert rel(got, 0.7 * OG.condensed_mul(op, G, x[:2 * N], N) - 0.4 * y[:2 * N]) <= 1e-12
    gz.op_fft.close()
