"""A Newton solve whose start already meets its tolerance takes no step, and its
direction is the start (zero for the predictor, the predictor's direction for
the corrector), whatever the buffers held before: with a relative tolerance of
2 nothing moves, and beta stays the soft-thresholded A'z0 the solve began
with, bit for bit.  The buffers are filled by an ADMM run first."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(4096,), (62, 82), (12, 10, 8)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("graphs", [False, True])
def test_no_step(cuda, size, precision, graphs):
    import csipm
    torch = cuda
    N = int(np.prod(size))
    rng = np.random.default_rng(N)
    keep = rng.random(N) > 0.2
    z0 = np.where(keep, rng.standard_normal(N), 0.0)
    params = csipm.FFTParameters(len(size), size, torch.tensor(z0, device="cuda"), 0.3, np.flatnonzero(~keep))
    nlp = csipm.FFTNLPModel(params, rdft=True, precision=precision, ipm_cg_rtol=2.0, max_iter=1, cuda_graphs=graphs)
    csipm.CompressedSensingADMM(params, nlp.op_fft, maxt=3)
    r = csipm.ipm_solve(nlp)
    assert r.stats["ipm_iter"] == 1 and r.stats["cg_iter"] == 0, r.stats
    b = nlp.M_perpt_z0
    want = torch.sign(b) * torch.clamp(b.abs() - 0.3, min=0.0)
    assert torch.equal(r.beta, want)
    nlp.op_fft.close()
