"""Norms of resident 1-D steps with weights of many decades."""
import numpy as np
import pytest

from tests.gpu_common import ensure_built

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def so():
    ensure_built()
    import split_operator_gb300 as so
    return so


# The state sits where the weights are 1e-9 of the largest: the loss at the border and the factor that
# restores the norm come from those weights.  Bounds of the resident lines over as many steps.
@pytest.mark.parametrize("precision,tol", [("fp64", 3e-14), ("float_float", 3e-13)])
@pytest.mark.parametrize("n", [64, 512, 500])
def test_resident_norms_with_weights_of_many_decades(so, precision, tol, n):
    from oracle import split_operator_oracle as O

    def build(lib):
        half = 20.0 * np.sqrt(n / 1024.0)
        x = -half + 2.0 * half / (n - 1.0) * np.arange(n)
        w = np.where(np.abs(x) < 0.8 * half, 1e-9, 1.0) * (x[1] - x[0])
        grid = lib.Grid.new_custom("space", x, w, 0)
        psi = np.exp(-(x / 0.4) ** 2 - 0.6j * x) * (np.abs(x) < 0.8 * half)
        wf = lib.WaveFunction(psi.astype(np.complex128), [grid])
        wf.normalize(1.0)
        tg = lib.TimeGrid(0.01, 10 ** 6)
        leak = lib.LeakControl()
        border = lib.BorderDumping((0.6 + 0.4 * np.cos(3.0 * x)).astype(np.complex128), grid)
        border.add_loss_checker(lib.LossChecker("border") if hasattr(lib, "LossChecker") else "border")
        st = lib.OperationStack()
        st.add_control(leak, lib.FIRST_HALF | lib.SECOND_HALF)
        st.add_control(border, lib.FIRST_HALF)
        st.add_propagator(lib.one_dim_into_propagator(0.5 * x * x, grid, tg, lib.HALF))
        st.add_transformation(lib.FFTTransformation(grid, "momentum"), lib.NORMAL)
        st.add_propagator(lib.one_dim_into_propagator(lib.kinetic_hamiltonian(grid, 1.0), grid, tg, lib.FULL))
        return wf, tg, st

    p = so.Propagation(*build(so), precision)
    q = O.Propagation(*build(O))
    p.set_timing(True)
    p.steps(1)
    q.propagate(1)
    assert "resident fx" in " ".join(k[0] for k in p.kernel_times())
    a, b = p.get_array(), q.wave_function.array
    assert np.linalg.norm(a - b) < tol * np.linalg.norm(b)
    assert abs(p.all_losses()[0] - q.all_losses()[0][1]) < tol
