"""Run-time-plan passes with the most stages their arguments hold: five stages
of a line, and rows one step past the tile (the in-place kernel).  FP64 against
the oracle (pocketfft) within 1e-12 relative."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def relerr(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


# rows of 1875 (3 5^4: five stages) and 6250 (in the tile), 6400 and 6402 (in
# place); strided lines of 1250 and 2000; 1D rows of 9375 and 46875
@pytest.mark.parametrize("size", [(3750, 4), (12500, 2), (12800, 2), (12804, 2), (4, 1250), (6, 2000),
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
