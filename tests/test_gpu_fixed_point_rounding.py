"""What lies below half a unit of a lane's fixed-point scale is rounded to zero, not to a unit of its
own sign, which would add up along a tail."""
import numpy as np
import pytest

from tests.gpu_common import ensure_built

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def so():
    ensure_built()
    import split_operator_gb300 as so
    return so


# A lane of one point and a tail of 1e-100 has the bits of the lane without the tail: each of its points
# rounds to zero.  (A unit per point, 2^-59 of the largest value, would make n 2^-59 of their sum.)
@pytest.mark.parametrize("n", [1000, 1024, 4096, 8192])
def test_a_tail_below_the_unit_adds_nothing(so, n):
    a = np.zeros((4, n), dtype=np.complex128)
    a[1], a[2], a[3] = 1e-100, -1e-100, 1e-30j
    a[:, n // 3] = 1.0
    lg = so.Grid.new_linear_countable("lane", 0.0, 3.0, 4, 0)
    xg = so.Grid.new_linear_continuos("x", -5.0, 5.0, n, 1)
    tg = so.TimeGrid(0.01, 100)
    st = so.OperationStack()
    st.add_transformation(so.FFTTransformation(xg, "k"), so.NORMAL)
    st.add_propagator(so.one_dim_into_propagator(so.kinetic_hamiltonian(xg, 1.0), xg, tg, so.FULL))
    p = so.Propagation(so.WaveFunction(a, [lg, xg]), tg, st, "fp64")
    p.set_timing(True)
    p.steps(1)
    assert "fftpair fx" in " ".join(k[0] for k in p.kernel_times())
    got = p.get_array()
    for row in got[1:]:
        np.testing.assert_array_equal(row, got[0])


@pytest.mark.parametrize("n", [64, 500, 512])
def test_a_tail_of_a_resident_line_adds_nothing(so, n):
    def run(tail):
        a = np.full(n, tail, dtype=np.complex128)
        a[n // 3] = 1.0
        xg = so.Grid.new_linear_continuos("x", -5.0, 5.0, n, 0)
        tg = so.TimeGrid(0.01, 100)
        st = so.OperationStack()
        st.add_transformation(so.FFTTransformation(xg, "k"), so.NORMAL)
        st.add_propagator(so.one_dim_into_propagator(so.kinetic_hamiltonian(xg, 1.0), xg, tg, so.FULL))
        p = so.Propagation(so.WaveFunction(a, [xg]), tg, st, "fp64")
        p.set_timing(True)
        p.steps(1)
        assert "resident fx" in " ".join(k[0] for k in p.kernel_times())
        return p.get_array()

    np.testing.assert_array_equal(run(1e-100), run(0.0))
