"""The norms inside resident 1-D steps are as accurate as FP64's: a step that loses part of its norm at a
border and is scaled back by a LeakControl has the scale of the same step in numpy."""
import numpy as np
import pytest

from tests.gpu_common import ensure_built

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def so():
    ensure_built()
    import split_operator_gb300 as so
    return so


def _line(lib, n, outer):
    half = 20.0 * np.sqrt(n / 1024.0)
    x = -half + 2.0 * half / (n - 1.0) * np.arange(n)
    w = np.where(np.abs(x) < 0.5 * half, 1.0, outer) * (x[1] - x[0])
    grid = lib.Grid.new_custom("space", x, w, 0)
    psi = np.exp(-(x / (0.3 * half)) ** 2 - 0.6j * x)
    wf = lib.WaveFunction(psi.astype(np.complex128), [grid])
    wf.normalize(1.0)
    tg = lib.TimeGrid(0.001, 10 ** 6)
    st = lib.OperationStack()
    st.add_control(lib.LeakControl(), lib.FIRST_HALF | lib.SECOND_HALF)
    st.add_control(lib.BorderDumping((0.75 + 0.25 * np.cos(x)).astype(np.complex128), grid), lib.FIRST_HALF)
    st.add_transformation(lib.FFTTransformation(grid, "momentum"), lib.NORMAL)
    st.add_propagator(lib.one_dim_into_propagator(lib.kinetic_hamiltonian(grid, 1.0), grid, tg, lib.FULL))
    return wf, tg, st


# numpy's two norms and the step's two, each within 2^-53 times a few (sums of squares of one sign); the
# scale is the root of their ratio: 2e-15 holds all of it
@pytest.mark.parametrize("outer", [1.0, 3.0, 60.0])
@pytest.mark.parametrize("n", [18, 64, 100, 300, 500, 512, 1000, 1024, 2046, 2048])
def test_the_scale_of_a_step_matches_numpy(so, n, outer):
    from oracle import split_operator_oracle as O
    p = so.Propagation(*_line(so, n, outer), "fp64")
    q = O.Propagation(*_line(O, n, outer))
    p.set_timing(True)
    p.steps(1)
    q.propagate(1)
    assert "resident fx" in " ".join(k[0] for k in p.kernel_times())
    a, b = p.get_array(), q.wave_function.array
    assert abs(np.vdot(b, a) / np.vdot(b, b) - 1.0) < 2e-15
