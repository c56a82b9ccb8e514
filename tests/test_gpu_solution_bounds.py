"""The c half of a solution [beta; c] (csipm_solve's c_out): c bounds |beta|, so
it is the same whichever order the solve keeps its vectors in, and carries none
of the signs the solver order folds into mirrored pairs.

Bounds: c - |beta| is a slack, positive up to the rounding of some tens of steps
(1e-15 of the largest entry each); the two orders' c at the repository's bound
for beta between configurations, 1e-6 relative."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


# 3D: every parity of the half sides, with and without a two-level pair along dim 2
@pytest.mark.parametrize("kind,dims", [("1d", (500,)), ("2d", (44, 62)), ("3d", (8, 6, 4)), ("3d", (14, 34, 22)),
                                       ("3d", (16, 32, 24)), ("3d", (26, 22, 36))],
                         ids=lambda v: v if isinstance(v, str) else "x".join(map(str, v)))
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_c_bounds_beta_in_both_orders(cuda, kind, dims, precision):
    import csipm
    import csipm.problems as P
    torch = cuda
    op0 = O.Operator(dims)
    prob = P.finalize(P.make_spec(kind, dims=dims, seed=4), op0.A, op0.At)
    got = {}
    for layout in ("solver", "reference"):
        params = csipm.FFTParameters(len(dims), dims, torch.tensor(prob.z0, device="cuda"), prob.lam, prob.missing)
        nlp = csipm.FFTNLPModel(params, rdft=True, precision=precision, tol=1e-10, ipm_cg_rtol=1e-2, layout=layout)
        r = csipm.ipm_solve(nlp)
        assert r.status == 0, r.stats
        n = nlp.nbeta
        beta, c = r.solution[:n].cpu().numpy(), r.solution[n:].cpu().numpy()
        assert np.all(c >= np.abs(beta) - 1e-9 * np.abs(beta).max())
        got[layout] = c
        nlp.op_fft.close()
    assert np.linalg.norm(got["solver"] - got["reference"]) <= 1e-6 * np.linalg.norm(got["reference"])
