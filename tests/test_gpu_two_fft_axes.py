"""Planes with an FFT on both axes: the pass along the contiguous axis that closes one step opens the
next ([inverse FFT, V/2, V/2, FFT, K]), FP64 and float-float."""
import numpy as np
import pytest

from tests.gpu_common import ensure_built

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def so():
    ensure_built()
    import split_operator_gb300 as so
    return so


def _stack(lib, nx, ny, seed):
    rng = np.random.default_rng(seed)
    xg = lib.Grid.new_linear_continuos("x", -8.0, 8.0, nx, 0)
    yg = lib.Grid.new_linear_continuos("y", -6.0, 6.0, ny, 1)
    x, y = np.asarray(xg.nodes)[:, None], np.asarray(yg.nodes)[None, :]
    psi = np.exp(-(x - 1.0) ** 2 - 0.5 * (y + rng.uniform(0.0, 0.5)) ** 2 + 0.8j * x - 0.3j * y)
    tg = lib.TimeGrid(0.01, 100)
    st = lib.OperationStack()
    st.add_propagator(lib.n_dim_into_propagator(0.5 * x * x + 0.7 * y * y + 0.1 * x * y, tg, lib.HALF))
    st.add_transformation(lib.FFTTransformation(xg, "kx"), lib.NORMAL)
    st.add_propagator(lib.one_dim_into_propagator(lib.kinetic_hamiltonian(xg, 1.0), xg, tg, lib.HALF))
    st.add_transformation(lib.FFTTransformation(yg, "ky"), lib.NORMAL)
    st.add_propagator(lib.one_dim_into_propagator(lib.kinetic_hamiltonian(yg, 1.0), yg, tg, lib.FULL))
    return lib.WaveFunction(psi.astype(np.complex128), [xg, yg]), tg, st


# four transforms a step, each within 5e-16 (float-float 2e-14 a stored pass), over 6 steps
@pytest.mark.parametrize("precision,tol", [("fp64", 3e-14), ("float_float", 5e-13)])
@pytest.mark.parametrize("nx,ny", [(512, 12), (1024, 38), (4096, 6), (256, 64), (300, 20)])
def test_two_fft_axes_match_the_oracle(so, precision, tol, nx, ny):
    from oracle import split_operator_oracle as O
    p = so.Propagation(*_stack(so, nx, ny, nx + ny), precision)
    q = O.Propagation(*_stack(O, nx, ny, nx + ny))
    p.set_timing(True)
    p.steps(6)
    q.propagate(6)
    names = [k[0] for k in p.kernel_times()]
    if precision == "float_float" and nx in (512, 1024, 4096):
        # the float-float pair kernel takes a transform pair in either order
        assert any("fftpair" in s and s.count("fft") >= 3 for s in names), names
    a, b = p.get_array(), q.wave_function.array
    assert np.linalg.norm(a - b) < tol * np.linalg.norm(b)


@pytest.mark.parametrize("precision", ["fp64", "float_float"])
def test_two_fft_axes_do_not_depend_on_the_split(so, precision):
    """Each pass computes on stored values alone; a run in parts stores once more at a step's end, in
    the same precision."""
    whole = so.Propagation(*_stack(so, 512, 12, 1), precision)
    whole.steps(4)
    parts = so.Propagation(*_stack(so, 512, 12, 1), precision)
    for k in (1, 3):
        parts.steps(k)
    a, b = whole.get_array(), parts.get_array()
    assert np.linalg.norm(a - b) < {"fp64": 1e-14, "float_float": 1e-13}[precision] * np.linalg.norm(a)
