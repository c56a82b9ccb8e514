"""Batches of recoveries whose rows run in place (longer than an on-chip tile):
refused as a batch before anything runs, solved one by one."""
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _problems(dims):
    import csipm.problems as P
    op0 = O.Operator(dims)
    return [P.finalize(P.make_spec("2d", dims=dims, seed=60 + k), op0.A, op0.At) for k in range(2)]


def _model(torch, prob):
    import csipm
    params = csipm.FFTParameters(2, prob.size, torch.tensor(prob.z0, device="cuda"), prob.lam, prob.missing)
    return csipm.FFTNLPModel(params, rdft=True, tol=1e-8, ipm_cg_rtol=1e-2)


# half rows of 6561 = 3^8 (8 stages in place) and 6480 (7)
@pytest.mark.parametrize("dims", [(13122, 4), (12960, 6)], ids=lambda s: "x".join(map(str, s)))
def test_batch_refuses_in_place_rows(cuda, dims):
    import csipm
    from csipm import _native
    torch = cuda
    models = [_model(torch, p) for p in _problems(dims)]
    with pytest.raises(_native.CsipmError) as e:
        csipm.ipm_solve_batch(models)
    assert e.value.status == _native.CSIPM_ERR_UNSUPPORTED and "solve it alone" in str(e.value)
    for m in models:
        r = csipm.ipm_solve(m)
        assert r.status == 0, r.stats
        m.op_fft.close()


def test_server_solves_them_one_by_one(cuda):
    """A batching server gets such requests solved all the same: equal to the
    solve alone (deterministic kernels), never an unsolved buffer with status 0."""
    from csipm.serving import Server
    import csipm
    torch = cuda
    dims = (13122, 4)
    probs = _problems(dims)
    with Server(slots=1, batch=4) as srv:
        for k in range(3):   # the first keeps the one slot busy while the others queue
            p = probs[k % 2]
            srv.submit(p.size, p.z0, p.lam, p.missing, tag=k, tol=1e-8, ipm_cg_rtol=1e-2)
        got = {r.tag: r for r in srv.drain()}
    for k in range(3):
        assert got[k].status == 0 and got[k].group == 1, got[k].message
        m = _model(torch, probs[k % 2])
        b = csipm.ipm_solve(m).beta.cpu().numpy()
        assert abs(got[k].beta - b).max() <= 1e-12 * abs(b).max()
        m.op_fft.close()
