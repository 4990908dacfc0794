"""Resident 1-D steps of a state of zeros: zeros come out, and a normalisation of it is reported as in
floating point."""
import numpy as np
import pytest

from tests.gpu_common import ensure_built

pytestmark = pytest.mark.gpu


def _line(so, n, leak, im):
    grid = so.Grid.new_linear_continuos("x", -5.0, 5.0, n, 0)
    tg = so.TimeGrid(0.01, 100, im)
    st = so.OperationStack()
    if leak:
        st.add_control(so.LeakControl(), so.FIRST_HALF | so.SECOND_HALF)
    st.add_propagator(so.one_dim_into_propagator(np.linspace(-1.0, 1.0, n) ** 2, grid, tg, so.HALF))
    st.add_transformation(so.FFTTransformation(grid, "k"), so.NORMAL)
    st.add_propagator(so.one_dim_into_propagator(so.kinetic_hamiltonian(grid, 1.0), grid, tg, so.FULL))
    p = so.Propagation(so.WaveFunction(np.zeros(n, dtype=np.complex128), [grid]), tg, st, "fp64")
    p.set_timing(True)
    return p


@pytest.mark.parametrize("im", [False, True])
@pytest.mark.parametrize("n", [64, 500, 512, 2048])
def test_a_zero_state_stays_zero(n, im):
    ensure_built()
    import split_operator_gb300 as so
    p = _line(so, n, False, im)
    p.steps(3)
    assert "resident fx" in " ".join(k[0] for k in p.kernel_times())
    assert np.all(p.get_array() == 0.0) and p.norm() == 0.0
    a = np.zeros(n, dtype=np.complex128)
    a[n - 1] = 1.0  # and the state that follows it is an ordinary one
    p.set_array(a)
    p.steps(1)
    unit = 1.0 if im else 1j
    v = np.exp(-unit * 0.005 * np.linspace(-1.0, 1.0, n) ** 2)
    kin = so.kinetic_hamiltonian(so.Grid.new_linear_continuos("x", -5.0, 5.0, n, 0), 1.0)
    ref = np.fft.ifft(np.fft.fft(a * v) * np.exp(-unit * 0.01 * np.asarray(kin))) * v
    assert np.linalg.norm(p.get_array() - ref) < 5e-15  # as a pair of transforms alone, of a norm of one


@pytest.mark.parametrize("n", [64, 500, 512])
def test_normalising_a_zero_state_is_reported(monkeypatch, n):
    ensure_built()
    import split_operator_gb300 as so
    from split_operator_gb300._lib import SplitOperatorError
    seen = []
    for fx in ("1", "0"):
        monkeypatch.setenv("SO_FX", fx)
        p = _line(so, n, True, False)
        p.steps(2)
        with pytest.raises(SplitOperatorError) as e:
            p.synchronize()
        seen.append((e.value.args, bool(np.all(np.isnan(p.get_array().real)))))
    assert seen[0] == seen[1]
