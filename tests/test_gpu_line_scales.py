"""Several normalisations in one resident 1-D step: the fixed-point values keep their headroom and their
bits through all of the factors."""
import numpy as np
import pytest

from tests.gpu_common import ensure_built

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def so():
    ensure_built()
    import split_operator_gb300 as so
    return so


def _line(lib, n, depth):
    half = 20.0 * np.sqrt(n / 1024.0)
    # weights that rise towards the outer half: a border there changes the norm and hardly the values
    x = -half + 2.0 * half / (n - 1.0) * np.arange(n)
    w = np.where(np.abs(x) < 0.5 * half, 1.0, 60.0) * (x[1] - x[0])
    grid = lib.Grid.new_custom("space", x, w, 0)
    psi = np.exp(-(x / (0.4 * half)) ** 2 - 0.6j * x)
    wf = lib.WaveFunction(psi.astype(np.complex128), [grid])
    wf.normalize(1.0)
    tg = lib.TimeGrid(0.001, 10 ** 6)
    st = lib.OperationStack()
    for _ in range(3):
        st.add_control(lib.LeakControl(), lib.FIRST_HALF | lib.SECOND_HALF)
        st.add_control(lib.BorderDumping(np.where(np.abs(x) < 0.5 * half, 1.0, depth).astype(np.complex128), grid),
                       lib.FIRST_HALF)
    st.add_transformation(lib.FFTTransformation(grid, "momentum"), lib.NORMAL)
    st.add_propagator(lib.one_dim_into_propagator(lib.kinetic_hamiltonian(grid, 1.0), grid, tg, lib.FULL))
    return wf, tg, st


# factors of a step together from 1.05 to 3: the bounds of the resident lines over 5 steps
@pytest.mark.parametrize("precision,tol", [("fp64", 3e-14), ("float_float", 3e-13)])
@pytest.mark.parametrize("depth", [0.97, 0.8, 0.6])
@pytest.mark.parametrize("n", [64, 500, 512])
def test_steps_with_three_leak_controls_match_the_oracle(so, precision, tol, n, depth):
    from oracle import split_operator_oracle as O
    p = so.Propagation(*_line(so, n, depth), precision)
    q = O.Propagation(*_line(O, n, depth))
    p.set_timing(True)
    p.steps(5)
    q.propagate(5)
    assert "resident fx" in " ".join(k[0] for k in p.kernel_times())
    a, b = p.get_array(), q.wave_function.array
    assert np.linalg.norm(a - b) < tol * np.linalg.norm(b)
    assert abs(p.norm() - q.wave_function.norm()) < tol
