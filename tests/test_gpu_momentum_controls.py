"""Controls behind the transformation of a resident 1-D step: their norms are taken on the momentum
grid, between the two transforms of the step, where the fixed-point values are not yet at the unitary
scale.  Every parity of log2 n, lengths that are no power of two, norms ahead of and behind the first
momentum-space factor, against the oracle.
"""
import numpy as np
import pytest

from tests.gpu_common import ensure_built

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def so():
    ensure_built()
    import split_operator_gb300 as so
    return so


def _checker(lib, name):
    return lib.LossChecker(name) if hasattr(lib, "LossChecker") else name


def _line(lib, n, kind, im):
    half = 20.0 * np.sqrt(n / 1024.0)
    grid = lib.Grid.new_linear_continuos("space", -half, half, n, 0)
    x = np.asarray(grid.nodes)
    psi = np.exp(-((x - 0.3 * half) / 1.7) ** 2 - 0.6j * x)
    wf = lib.WaveFunction(psi.astype(np.complex128), [grid])
    wf.normalize(1.0)
    tg = lib.TimeGrid(0.01, 10 ** 6, im)
    both = lib.FIRST_HALF | lib.SECOND_HALF
    leak = lib.LeakControl()
    # factors of 0.3 to 1 on the momentum grid, in FFT order
    border = lib.BorderDumping((0.65 + 0.35 * np.cos(2.0 * np.pi * np.arange(n) / n)).astype(np.complex128), grid)
    border.add_loss_checker(_checker(lib, "border"))
    kin = lib.one_dim_into_propagator(lib.kinetic_hamiltonian(grid, 1.0), grid, tg, lib.FULL)
    st = lib.OperationStack()
    st.add_propagator(lib.one_dim_into_propagator(0.5 * x * x, grid, tg, lib.HALF))
    st.add_transformation(lib.FFTTransformation(grid, "momentum"), lib.NORMAL)
    if kind == "after":  # every norm behind a factor
        st.add_propagator(kin)
        st.add_control(border, both)
    else:
        if kind in ("leak", "leak_border"):
            st.add_control(leak, both)
        if kind in ("border", "leak_border"):
            st.add_control(border, both)
        st.add_propagator(kin)
    return wf, tg, st


# the bounds of the resident lines' own test: 30 steps of numpy's FP64 against as many fixed-point ones
@pytest.mark.parametrize("precision,tol", [("fp64", 3e-14), ("float_float", 3e-13)])
@pytest.mark.parametrize("kind", ["leak", "border", "leak_border", "after"])
@pytest.mark.parametrize("n,im", [(n, False) for n in (16, 32, 64, 256, 500, 512, 1024, 2048)] +
                         [(n, True) for n in (64, 500, 512)])
def test_controls_in_momentum_space_match_the_oracle(so, precision, tol, kind, n, im):
    from oracle import split_operator_oracle as O
    p = so.Propagation(*_line(so, n, kind, im), precision)
    q = O.Propagation(*_line(O, n, kind, im))
    p.set_timing(True)
    p.steps(30)
    q.propagate(30)
    assert "resident fx" in " ".join(k[0] for k in p.kernel_times())
    a, b = p.get_array(), q.wave_function.array
    assert np.linalg.norm(a - b) < tol * np.linalg.norm(b)
    assert abs(p.norm() - q.wave_function.norm()) < tol * max(1.0, q.wave_function.norm())
    got, ref = p.all_losses(), [v for _, v in q.all_losses()]
    assert len(got) == len(ref) and np.abs(np.array(got) - np.array(ref)).max(initial=0.0) < 30 * tol
