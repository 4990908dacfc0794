"""Full-size tables at the limit of the device's memory: the scratch copy of a table's upload and the
fixed-point copy of a table are taken only where there is room, and the passes run without them."""
import numpy as np
import pytest

from tests.gpu_common import ensure_built

pytestmark = pytest.mark.gpu


def _build(so, n, nq, nr):
    x, w = np.polynomial.legendre.leggauss(n)
    v = np.stack([np.sqrt(l + 0.5) * np.polynomial.legendre.Legendre.basis(l)(x) for l in range(n)])
    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, nq, nr)) + 1j * rng.standard_normal((n, nq, nr))
    ph = np.exp(1j * rng.uniform(0.0, 6.0, (n, nq, nr)))
    pg = so.Grid.new_linear_countable("p", 0.0, n - 1.0, n, 0)
    qg = so.Grid.new_linear_countable("q", 0.0, nq - 1.0, nq, 1)
    rg = so.Grid.new_linear_countable("r", 0.0, nr - 1.0, nr, 2)
    st = so.OperationStack()
    mt = so.MatrixTransformation(pg, so.Grid.new_linear_countable("l", 0.0, n - 1.0, n, 0))
    mt.set_diagonalization_matrix(v * w[None, :], v.T.copy())
    st.add_transformation(mt, so.NORMAL)
    pd = so.NDimPropagator()
    pd.set_operator(ph)
    st.add_propagator(pd)
    wf = so.WaveFunction(a, [pg, qg, rg])
    p = so.Propagation(wf, so.TimeGrid(0.01, 100), st, "fp64")
    p.set_timing(True)

    def step(r):  # [T, phase, T^-1] at the points r of the last axis
        return np.einsum("lp,lqr->pqr", v, np.einsum("lp,pqr->lqr", v * w[None, :], a[:, :, r]) * ph[:, :, r])

    return p, wf, step


# Room for the source state, the propagation's and the table, and beside them for
#  half an array: no scratch copy for the upload (the host orders the table), no fixed-point copy;
#  an array and a half: no fixed-point copy, as that would take the room of the state's copy in mean_energy
@pytest.mark.parametrize("beside", [0.5, 1.5])
def test_tables_without_room_for_their_copies(beside):
    ensure_built()
    import torch

    import split_operator_gb300 as so
    n, nq, nr = 64, 128, 2048
    array = n * nq * nr * 16  # 268 MB
    for env in ("1", "0"):  # the kernels of both routes are loaded
        with pytest.MonkeyPatch.context() as m:
            m.setenv("SO_FX", env)
            q, *_ = _build(so, n, 2, 64)
            q.steps(1)
            q.mean_energy()
            del q
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    hold = torch.empty(free - int((3 + beside) * array), dtype=torch.uint8, device="cuda")
    try:
        p, wf, step = _build(so, n, nq, nr)
        p.steps(1)
        assert "tcfx" not in " ".join(k[0] for k in p.kernel_times())
        if beside > 1:
            p.mean_energy()  # (one more step)
    finally:
        del hold
        torch.cuda.empty_cache()
    if beside < 1:
        some = np.arange(5, nr, 97)
        np.testing.assert_allclose(p.get_array()[:, :, some], step(some), rtol=0.0, atol=1e-12)
    # with room again, a new propagation takes the fixed-point pass
    r, *_ = _build(so, n, nq, nr)
    r.steps(1 if beside < 1 else 2)
    assert "tcfx" in " ".join(k[0] for k in r.kernel_times())
    got = p.get_array()
    assert np.linalg.norm(r.get_array() - got) < 2e-14 * np.linalg.norm(got)


def test_an_out_of_memory_error_ends_with_its_call():
    ensure_built()
    import torch

    import split_operator_gb300 as so
    p, wf, step = _build(so, 64, 2, 64)
    p.steps(1)
    torch.cuda.empty_cache()
    hold = torch.empty(torch.cuda.mem_get_info()[0] - (1 << 28), dtype=torch.uint8, device="cuda")
    try:
        with pytest.raises(Exception, match="out of memory"):
            so.WaveFunction(np.zeros((1 << 15, 1 << 10), dtype=np.complex128),  # 512 MB
                            [so.Grid.new_linear_countable("a", 0.0, 1.0, 1 << 15, 0),
                             so.Grid.new_linear_countable("b", 0.0, 1.0, 1 << 10, 1)])
        p.steps(1)
    finally:
        del hold
        torch.cuda.empty_cache()
    q, *_ = _build(so, 64, 2, 64)
    q.steps(2)
    np.testing.assert_array_equal(p.get_array(), q.get_array())
