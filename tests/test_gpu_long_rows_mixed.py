"""Mixed-precision recoveries whose FP64 rows run in place while the FP32 rows
still take a tile (half rows of 6402 = 2 3 11 97 and 6561 = 3^8): against the FP64
solve at the bounds of the mixed-precision tests (beta 1e-6, objective 1e-8)."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(12804, 4), (13122, 6)], ids=lambda s: "x".join(map(str, s)))
def test_recovery(cuda, dims):
    import csipm
    import csipm.problems as P
    torch = cuda
    op0 = O.Operator(dims)
    prob = P.finalize(P.make_spec("2d", dims=dims, seed=7), op0.A, op0.At)
    got = {}
    for precision in ("fp64", "mixed"):
        params = csipm.FFTParameters(2, dims, torch.tensor(prob.z0, device="cuda"), prob.lam, prob.missing)
        nlp = csipm.FFTNLPModel(params, rdft=True, precision=precision, tol=1e-10, ipm_cg_rtol=1e-2)
        r = csipm.ipm_solve(nlp)
        assert r.status == 0, r.stats
        got[precision] = (r.beta.cpu().numpy(), r.stats["lasso_obj"])
        nlp.op_fft.close()
    (b64, f64), (b32, f32) = got["fp64"], got["mixed"]
    assert np.linalg.norm(b32 - b64) <= 1e-6 * np.linalg.norm(b64)
    assert abs(f32 - f64) <= 1e-8 * abs(f64)
