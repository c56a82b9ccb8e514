"""Short 1D rows, whose products run in one launch (l1d_one_kernel,
csrc/long1d.cuh), and the first size above them: smallest rows, odd and prime half
lengths, with and without missing samples, against the oracle within 1e-12."""
import ctypes

import numpy as np
import pytest

import oracle as O
import oracle_ipm as OI

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


# half lengths 1, 2, 3, 11, 31, 64, 5 5 5 7, 1021 (prime), 23 89, 2048, 3 683
@pytest.mark.parametrize("N", [2, 4, 6, 22, 62, 128, 1750, 2042, 4094, 4096, 4098])
@pytest.mark.parametrize("masked", [True, False])
def test_products(cuda, N, masked):
    import csipm
    torch = cuda
    rng = np.random.default_rng(N)
    keep = rng.random(N) > 0.3 if masked else np.ones(N, dtype=bool)
    if masked:
        keep[0], keep[-1] = True, False   # one observed and one missing at least
    z0 = np.where(keep, rng.standard_normal(N), 0.0)
    params = csipm.FFTParameters(1, (N,), torch.tensor(z0, device="cuda"), 0.3, np.flatnonzero(~keep))
    nlp = csipm.FFTNLPModel(params, rdft=True)
    op, ref = nlp.op_fft, O.Operator((N,), keep)
    dev = lambda v: torch.tensor(v, device="cuda")
    x, y = rng.standard_normal(6 * N), rng.standard_normal(6 * N)
    xt = dev(x[:N])
    assert rel(op.M_perp_beta(xt).cpu().numpy(), ref.A(x[:N])) <= 1e-12
    assert rel(op.M_perpt_z(xt).cpu().numpy(), ref.At(x[:N])) <= 1e-12
    want = ref.AtA(x[:N])
    assert np.linalg.norm(op.M_perpt_M_perp_vec(xt).cpu().numpy() - want) <= 1e-12 * np.linalg.norm(x[:N])
    kkt = csipm.FFTKKTSystem(nlp)
    pr = np.ones(4 * N)
    pr[2 * N:] = rng.uniform(0.05, 20.0, 2 * N)
    kkt.build_kkt(dev(pr))
    K = OI.kkt_build(pr, N)
    got = kkt.condensed_mul(dev(y[:2 * N]), dev(x[:2 * N]), 0.7, -0.4).cpu().numpy()
    assert rel(got, OI.condensed_mul(ref, K, y[:2 * N], x[:2 * N], 0.7, -0.4)) <= 1e-12
    assert rel(kkt.mul(dev(y), dev(x), 0.7, -0.4).cpu().numpy(), OI.kkt_mul(ref, y, x, 0.7, -0.4)) <= 1e-12
    # the entry point without allocations
    bits = None
    if masked:
        padded = np.zeros((N + 31) // 32 * 32, dtype=np.uint8)
        padded[:N] = keep
        bits = torch.tensor(np.packbits(padded, bitorder="little").view(np.int32), device="cuda")
    out = torch.empty_like(xt)
    size = (ctypes.c_int * 3)(N, 1, 1)
    st = torch.cuda.current_stream().cuda_stream
    assert csipm.lib().csipm_apply_AtA_static(1, size, ctypes.c_void_p(bits.data_ptr() if masked else None),
                                              ctypes.c_void_p(xt.data_ptr()), ctypes.c_void_p(out.data_ptr()),
                                              ctypes.c_void_p(st)) == 0
    assert np.linalg.norm(out.cpu().numpy() - want) <= 1e-12 * np.linalg.norm(x[:N])
    op.close()


@pytest.mark.parametrize("N", [500, 2042, 4096])
def test_mixed_precision_recovery(cuda, N):
    """The FP32 instantiation: mixed against FP64 at the bounds of the
    mixed-precision tests (beta 1e-6, objective 1e-8)."""
    import csipm
    import csipm.problems as P
    torch = cuda
    op0 = O.Operator((N,))
    prob = P.finalize(P.make_spec("1d", dims=(N,), seed=8), op0.A, op0.At)
    got = {}
    for precision in ("fp64", "mixed"):
        params = csipm.FFTParameters(1, (N,), torch.tensor(prob.z0, device="cuda"), prob.lam, prob.missing)
        nlp = csipm.FFTNLPModel(params, rdft=True, precision=precision, tol=1e-10, ipm_cg_rtol=1e-2)
        r = csipm.ipm_solve(nlp)
        assert r.status == 0, r.stats
        got[precision] = (r.beta.cpu().numpy(), r.stats["lasso_obj"])
        nlp.op_fft.close()
    (b64, f64), (b32, f32) = got["fp64"], got["mixed"]
    assert rel(b32, b64) <= 1e-6 and abs(f32 - f64) <= 1e-8 * abs(f64)
