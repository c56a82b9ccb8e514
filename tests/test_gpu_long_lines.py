"""Run-time-plan passes with the most stages their arguments hold: five and six
stages of a line, and rows one step past the tile (the in-place kernel).  FP64
against the oracle (pocketfft) within 1e-12 relative; mixed precision against
the FP64 solve at the bounds of the mixed-precision tests."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def relerr(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


# rows of 1875 (3 5^4: five stages), 6250 and 6400 (the last that fit two FP64
# buffers), 6402 and 9375 (in place); lines of 1250, 1875 and 2000
@pytest.mark.parametrize("size", [(3750, 4), (12500, 2), (12800, 2), (12804, 2), (18750, 4), (4, 1250), (6, 2000),
                                  (2 * 9375,), (2 * 46875,)], ids=lambda s: "x".join(map(str, s)))
def test_products(cuda, size):
    import csipm
    torch = cuda
    N = int(np.prod(size))
    rng = np.random.default_rng(N)
    keep = rng.random(N) > 0.2
    z0 = np.where(keep, rng.standard_normal(N), 0.0)
    params = csipm.FFTParameters(len(size), size, torch.tensor(z0, device="cuda"), 0.1, np.flatnonzero(~keep))
    op = csipm.FFTNLPModel(params, rdft=True).op_fft
    ref = O.Operator(size, keep)
    x = rng.standard_normal(N)
    xt = torch.tensor(x, device="cuda")
    assert relerr(op.M_perp_beta(xt).cpu().numpy(), ref.A(x)) <= 1e-12
    assert relerr(op.M_perpt_z(xt).cpu().numpy(), ref.At(x)) <= 1e-12
    assert relerr(op.M_perpt_M_perp_vec(xt).cpu().numpy(), ref.AtA(x)) <= 1e-12
    op.close()


def test_six_stages_fp32(cuda):
    """Rows of 9375 = 3 5^5 values: six stages in one FP32 tile."""
    import csipm
    import csipm.problems as P
    torch = cuda
    dims = (18750, 26)
    op0 = O.Operator(dims)
    prob = P.finalize(P.make_spec("2d", dims=dims, seed=5), op0.A, op0.At)
    got = {}
    for precision in ("fp64", "mixed"):
        params = csipm.FFTParameters(2, dims, torch.tensor(prob.z0, device="cuda"), prob.lam, prob.missing)
        nlp = csipm.FFTNLPModel(params, rdft=True, precision=precision, tol=1e-10, ipm_cg_rtol=1e-2)
        r = csipm.ipm_solve(nlp)
        assert r.status == 0, r.stats
        got[precision] = (r.beta.cpu().numpy(), r.stats["lasso_obj"])
        nlp.op_fft.close()
    assert relerr(got["mixed"][0], got["fp64"][0]) <= 1e-6
    assert abs(got["mixed"][1] - got["fp64"][1]) <= 1e-8 * abs(got["fp64"][1])
