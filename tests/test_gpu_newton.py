"""solve_kkt! on N unknowns (csrc/solver_kernels.cuh): its iterates are those of
the 2N preconditioned CG, so a solve stopped early gives the 2N method's
iterate, not only its limit.  Against the numpy statement of the 2N method, in
both orders of the vectors.

Bound: both take the same steps in exact arithmetic; rounding enters at 1e-16
a step, grows at most with the preconditioned condition number (1 + 1e3 here)
over some 20 steps and the back-substitution's 1/S <= 1e2: 1e-9 relative."""
import numpy as np
import pytest

import oracle as O
import oracle_ipm as OI

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(200,), (4100,), (12, 18), (62, 82), (2, 6), (8, 6, 4), (22, 14, 34), (48, 44, 52)],
                         ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("rtol", [0.3, 1e-2, 1e-5, 1e-12])
@pytest.mark.parametrize("layout", ["solver", "reference"])
def test_iterates_of_the_2n_method(cuda, size, rtol, layout):
    import csipm
    torch = cuda
    N = int(np.prod(size))
    rng = np.random.default_rng(N)
    keep = rng.random(N) > 0.2
    z0 = np.where(keep, rng.standard_normal(N), 0.0)
    params = csipm.FFTParameters(len(size), size, torch.tensor(z0, device="cuda"), 0.3, np.flatnonzero(~keep))
    nlp = csipm.FFTNLPModel(params, rdft=True, cg_atol=0.0, cg_rtol=rtol, layout=layout)
    kkt = csipm.FFTKKTSystem(nlp)
    pr = np.ones(4 * N)
    pr[2 * N:] = 10.0 ** rng.uniform(-2.0, 2.0, 2 * N)
    prt = torch.tensor(pr, device="cuda")
    kkt.build_kkt(prt)
    w = rng.standard_normal(6 * N)
    wt = torch.tensor(w, device="cuda")
    kkt.solve_kkt(wt, prt)
    sol, it = OI.kkt_solve(O.Operator(size, keep), OI.kkt_build(pr, N), w, pr, atol=0.0, rtol=rtol)
    assert kkt.krylov_iterations[-1] == it or (rtol < 1e-10 and abs(kkt.krylov_iterations[-1] - it) <= 1)
    got = wt.cpu().numpy()
    assert np.linalg.norm(got - sol) <= 1e-9 * np.linalg.norm(sol)
    nlp.op_fft.close()


def test_zero_right_hand_side(cuda):
    """w = 0 stops before the first iteration."""
    import csipm
    torch = cuda
    n = 24 * 20
    params = csipm.FFTParameters(2, (24, 20), torch.ones(n, dtype=torch.float64, device="cuda"), 0.3, None)
    nlp = csipm.FFTNLPModel(params, rdft=True)
    kkt = csipm.FFTKKTSystem(nlp)
    pr = torch.ones(4 * n, dtype=torch.float64, device="cuda")
    kkt.build_kkt(pr)
    w = torch.zeros(6 * n, dtype=torch.float64, device="cuda")
    kkt.solve_kkt(w, pr)
    assert kkt.krylov_iterations == [0] and not w.any()
