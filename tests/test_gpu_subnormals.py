"""States whose values are below the smallest normal number: fixed-point passes keep them, to the
spacing of the subnormal numbers, as floating-point ones do."""
import numpy as np
import pytest

from tests.gpu_common import ensure_built

pytestmark = pytest.mark.gpu

# scale of the values, its inverse (a power of two: exact), and the spacing of the subnormal numbers
TINY = {"fp64": (2.0 ** -1030, 1030, 2.0 ** -1074), "float_float": (2.0 ** -133, 133, 2.0 ** -149)}


@pytest.fixture(scope="module")
def so():
    ensure_built()
    import split_operator_gb300 as so
    return so


def _up(a, e):
    """a 2^e without a factor out of range"""
    return np.ldexp(a.real, e) + 1j * np.ldexp(a.imag, e)


# the result is rounded once to the spacing; the transforms' own roundings, 2^-60 of the lane's norm or
# of the smallest exponent a lane is scaled by, stay below it: 8 spacings hold both
@pytest.mark.parametrize("precision", ["fp64", "float_float"])
@pytest.mark.parametrize("n", [16, 500, 512, 4096])
def test_fft_pair_of_subnormal_lanes(so, precision, n):
    tiny, e, unit = TINY[precision]
    rng = np.random.default_rng(n)
    a = np.round((rng.standard_normal((5, n)) + 1j * rng.standard_normal((5, n))) * 2.0 ** 14) * 2.0 ** -14
    a[1] = 0.0
    a[1, 3] = unit / tiny            # a single value of one spacing
    a[2] *= 2.0 ** 100                # a normal lane beside them
    a[3, ::2] *= 2.0 ** 12            # normal and subnormal values in one lane
    lg = so.Grid.new_linear_countable("lane", 0.0, 4.0, 5, 0)
    xg = so.Grid.new_linear_continuos("x", -5.0, 5.0, n, 1)
    tg = so.TimeGrid(1e-6, 100)
    st = so.OperationStack()
    st.add_transformation(so.FFTTransformation(xg, "k"), so.NORMAL)
    kin = so.kinetic_hamiltonian(xg, 1.0)
    st.add_propagator(so.one_dim_into_propagator(kin, xg, tg, so.FULL))
    p = so.Propagation(so.WaveFunction(_up(a, -e), [lg, xg]), tg, st, precision)
    p.set_timing(True)
    p.steps(1)
    assert "fftpair fx" in " ".join(k[0] for k in p.kernel_times())
    got = _up(p.get_array(), e)
    ref = np.fft.ifft(np.fft.fft(a, axis=1) * np.exp(-1e-6j * kin), axis=1)
    rel = {"fp64": 2e-15, "float_float": 2e-14}[precision]
    for l in range(5):
        err = np.abs(got[l] - ref[l]).max()
        assert err <= 8 * unit / tiny + rel * np.linalg.norm(ref[l]), (l, err * tiny / unit)
        assert np.any(got[l] != 0.0) or l == 1


@pytest.mark.parametrize("precision", ["fp64", "float_float"])
@pytest.mark.parametrize("n,nr", [(32, 40), (200, 9)])
def test_lane_matrices_on_subnormal_columns(so, precision, n, nr):
    tiny, e, unit = TINY[precision]
    rng = np.random.default_rng(n)
    x, w = np.polynomial.legendre.leggauss(n)
    v = np.stack([np.sqrt(l + 0.5) * np.polynomial.legendre.Legendre.basis(l)(x) for l in range(n)])
    t, tinv = v * w[None, :], v.T.copy()
    a = np.round((rng.standard_normal((n, nr)) + 1j * rng.standard_normal((n, nr))) * 2.0 ** 14) * 2.0 ** -14
    a[:, 1] *= 2.0 ** 100
    a[::2, 2] *= 2.0 ** 12

    def build():
        pg = so.Grid.new_linear_countable("p", 0.0, n - 1.0, n, 0)
        rg = so.Grid.new_linear_continuos("r", 0.0, 5.0, nr, 1)
        st = so.OperationStack()
        mt = so.MatrixTransformation(pg, so.Grid.new_linear_countable("l", 0.0, n - 1.0, n, 0))
        mt.set_diagonalization_matrix(t, tinv)
        st.add_transformation(mt, so.NORMAL)
        pd = so.NDimPropagator()
        pd.set_operator(ph)
        st.add_propagator(pd)
        return so.Propagation(so.WaveFunction(_up(a, -e), [pg, rg]), so.TimeGrid(0.01, 100), st, precision)

    ph = np.exp(1j * rng.uniform(0.0, 6.0, (n, nr)))
    p = build()
    p.set_timing(True)
    p.steps(1)
    assert "tcfx" in " ".join(k[0] for k in p.kernel_times())
    got, ref = _up(p.get_array(), e), tinv @ ((t @ a) * ph)
    rel = {"fp64": 4e-15, "float_float": 8e-14}[precision]
    err = np.abs(got - ref).max(axis=0)
    assert np.all(err <= 2 * unit / tiny + rel * np.linalg.norm(ref, axis=0)), err.max() * tiny / unit
    # a step's end inside a pass keeps the 53 bits that a store rounds to the spacing: two such stores
    # more in the run in parts, through orthonormal transforms
    whole, parts = build(), build()
    whole.steps(4)
    for k in (1, 2, 1):
        parts.steps(k)
    diff = np.linalg.norm(_up(whole.get_array(), e) - _up(parts.get_array(), e), axis=0)
    assert np.all(diff <= 2 * np.sqrt(2 * n) * unit / tiny + rel * np.linalg.norm(ref, axis=0))
    assert np.all(np.any(whole.get_array() != 0.0, axis=0))


@pytest.mark.parametrize("precision", ["fp64", "float_float"])
@pytest.mark.parametrize("n", [16, 500, 1024])
def test_resident_line_of_a_subnormal_state(so, precision, n):
    tiny, e, unit = TINY[precision]
    rng = np.random.default_rng(n)
    a = np.round((rng.standard_normal(n) + 1j * rng.standard_normal(n)) * 2.0 ** 14) * 2.0 ** -14
    grid = so.Grid.new_linear_continuos("x", -5.0, 5.0, n, 0)
    tg = so.TimeGrid(1e-6, 100)
    st = so.OperationStack()
    st.add_transformation(so.FFTTransformation(grid, "k"), so.NORMAL)
    kin = so.kinetic_hamiltonian(grid, 1.0)
    st.add_propagator(so.one_dim_into_propagator(kin, grid, tg, so.FULL))
    p = so.Propagation(so.WaveFunction(_up(a, -e), [grid]), tg, st, precision)
    p.set_timing(True)
    p.steps(1)
    assert "resident fx" in " ".join(k[0] for k in p.kernel_times())
    got = _up(p.get_array(), e)
    ref = np.fft.ifft(np.fft.fft(a) * np.exp(-1e-6j * kin))
    assert np.abs(got - ref).max() <= 8 * unit / tiny + 2e-14 * np.linalg.norm(ref)
    assert np.any(got != 0.0)
