"""Iterations that leave the usual path of csipm_solve: mixed-precision Newton
solves whose FP32 CG overflows (finished in FP64), and iterations that a graph
replay hands back to the host because a CG loop reached its cap.  Both against
the FP64 solve at the bounds of the mixed-precision tests (beta 1e-6)."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

SIZES = [("1d", (2000,)), ("2d", (64, 48)), ("3d", (16, 18, 20))]


def _solve(torch, prob, scale=1.0, **opts):
    import csipm
    params = csipm.FFTParameters(len(prob.size), prob.size, torch.tensor(prob.z0 * scale, device="cuda"),
                                 prob.lam * scale, prob.missing)
    nlp = csipm.FFTNLPModel(params, rdft=True, tol=1e-10, **opts)
    r = csipm.ipm_solve(nlp)
    out = r.status, r.beta.cpu().numpy() / scale, r.stats
    nlp.op_fft.close()
    return out


def _problem(kind, dims):
    import csipm.problems as P
    op0 = O.Operator(dims)
    return P.finalize(P.make_spec(kind, dims=dims, seed=9), op0.A, op0.At)


@pytest.mark.parametrize("kind,dims", SIZES)
@pytest.mark.parametrize("graphs", [True, False])
def test_fp32_overflow_is_finished_in_fp64(cuda, kind, dims, graphs):
    """z0 and lambda times 1e60 (the problem is homogeneous): no FP32 residual
    is finite, so every Newton solve falls back."""
    prob = _problem(kind, dims)
    opts = dict(ipm_cg_rtol=1e-6, cuda_graphs=graphs)
    s64, b64, _ = _solve(cuda, prob, 1e60, precision="fp64", **opts)
    s32, b32, st = _solve(cuda, prob, 1e60, precision="mixed", **opts)
    assert s64 == s32 == 0 and st["fallbacks"] == 2 * st["ipm_iter"] > 0
    assert np.linalg.norm(b32 - b64) <= 1e-6 * np.linalg.norm(b64)


@pytest.mark.parametrize("kind,dims", SIZES)
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_iterations_handed_back_by_a_replay(cuda, kind, dims, precision):
    prob = _problem(kind, dims)
    s64, b64, _ = _solve(cuda, prob, precision="fp64", ipm_cg_rtol=1e-3, cuda_graphs=False)
    s, b, st = _solve(cuda, prob, precision=precision, ipm_cg_rtol=1e-3, cg_maxit=2, cuda_graphs=True)
    assert s64 == s == 0
    if precision == "mixed":
        assert st["graph_iters"] < st["ipm_iter"]
    assert np.linalg.norm(b - b64) <= 1e-6 * np.linalg.norm(b64)
