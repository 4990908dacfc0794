"""Fixed-point passes whose factors differ by many decades from column to column (lane to lane): each
keeps its own relative accuracy."""
import numpy as np
import pytest

from tests.gpu_common import ensure_built

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def so():
    ensure_built()
    import split_operator_gb300 as so
    return so


def _legendre(n):
    x, w = np.polynomial.legendre.leggauss(n)
    v = np.stack([np.sqrt(l + 0.5) * np.polynomial.legendre.Legendre.basis(l)(x) for l in range(n)])
    return v * w[None, :], v.T.copy()


# Exponents of the factors from column to column (FP64: down to e^-60, four of them over two steps;
# float-float: within FP32's exponents)
DECAY = {"fp64": 60.0, "float_float": 15.0}
# the transforms' and the phase's 16 roundings of the lane-matrix test, and the factors' own: of each
# table value and of each product, four tables over two steps, 2^-53 (float-float 2^-47) each
MAT_TOL = {"fp64": 6e-15, "float_float": 2e-13}


@pytest.mark.parametrize("precision", ["fp64", "float_float"])
@pytest.mark.parametrize("kind", ["nd", "axis", "both"])
@pytest.mark.parametrize("n,nr", [(16, 8), (33, 41), (64, 700), (128, 33), (200, 40)])
def test_lane_matrix_columns_of_small_factors(so, precision, kind, n, nr):
    rng = np.random.default_rng(n + nr)
    t, tinv = _legendre(n)
    a = (rng.standard_normal((n, nr)) + 1j * rng.standard_normal((n, nr))).astype(np.complex64).astype(np.complex128)
    c = np.linspace(0.0, DECAY[precision], nr)
    c = rng.permutation(c)
    nd = np.exp(-c[None, :] * rng.uniform(0.97, 1.0, (n, nr)))
    axis = np.exp(-c)
    if kind == "both":
        nd, axis = np.sqrt(nd), np.sqrt(axis)
    nd[:, nr // 2] = 0.0
    axis[nr // 2] = 0.0
    ph = np.exp(1j * rng.uniform(0.0, 6.0, (n, nr)))
    pg = so.Grid.new_linear_countable("p", 0.0, n - 1.0, n, 0)
    rg = so.Grid.new_linear_continuos("r", 0.0, 5.0, nr, 1)
    st = so.OperationStack()
    if kind != "axis":
        d = so.NDimPropagator()
        d.set_operator(nd.astype(np.complex128))
        st.add_propagator(d)
    if kind != "nd":
        d = so.OneDimPropagator(nr, 1)
        d.set_operator(axis.astype(np.complex128))
        st.add_propagator(d)
    mt = so.MatrixTransformation(pg, so.Grid.new_linear_countable("l", 0.0, n - 1.0, n, 0))
    mt.set_diagonalization_matrix(t, tinv)
    st.add_transformation(mt, so.NORMAL)
    d = so.NDimPropagator()
    d.set_operator(ph)
    st.add_propagator(d)
    p = so.Propagation(so.WaveFunction(a, [pg, rg]), so.TimeGrid(0.01, 100), st, precision)
    p.set_timing(True)
    p.steps(2)
    assert "tcfx" in " ".join(k[0] for k in p.kernel_times())

    def mul(m, z):
        m = m.real.astype(np.longdouble)
        return m @ z.real.astype(np.longdouble) + 1j * (m @ z.imag.astype(np.longdouble))

    f = np.ones((n, nr), dtype=np.longdouble)
    if kind != "axis":
        f = f * nd
    if kind != "nd":
        f = f * axis[None, :]
    ref = a.astype(np.clongdouble)
    for _ in range(2):
        ref = mul(tinv, mul(t, ref * f) * ph) * f
    got = p.get_array()
    assert np.all(got[:, nr // 2] == 0.0)
    live = np.arange(nr) != nr // 2
    scale = np.abs(ref).max(axis=0)[live].astype(np.longdouble)
    err = np.linalg.norm(((got - ref)[:, live] / scale).astype(np.complex128), axis=0)
    err /= np.linalg.norm((ref[:, live] / scale).astype(np.complex128), axis=0)
    assert err.max() < MAT_TOL[precision], (int(err.argmax()), err.max())


# numpy's pair and the fixed-point one within 5e-16 and 4e-16, the table after it two roundings
LANE_TOL = {"fp64": 3e-15, "float_float": 3e-14}


@pytest.mark.parametrize("precision", ["fp64", "float_float"])
@pytest.mark.parametrize("n,lanes", [(16, 70), (256, 37), (1000, 9), (2048, 5), (8192, 3)])
def test_fft_pair_lanes_of_small_factors(so, precision, n, lanes):
    rng = np.random.default_rng(n)
    a = rng.standard_normal((lanes, n)) + 1j * rng.standard_normal((lanes, n))
    c = np.linspace(0.0, DECAY[precision], lanes)
    t = np.exp(-c[:, None] * rng.uniform(0.97, 1.0, (lanes, n)) - 1j * rng.uniform(-3.0, 3.0, (lanes, n)))
    lg = so.Grid.new_linear_countable("lane", 0.0, lanes - 1.0, lanes, 0)
    xg = so.Grid.new_linear_continuos("x", -5.0, 5.0, n, 1)
    tg = so.TimeGrid(0.01, 100)
    st = so.OperationStack()
    # an identity along the lane axis keeps the table before the transforms in a pass of its own
    mt = so.MatrixTransformation(lg, so.Grid.new_linear_countable("same", 0.0, lanes - 1.0, lanes, 0))
    mt.set_diagonalization_matrix(np.eye(lanes), np.eye(lanes))
    st.add_transformation(mt, so.NORMAL)
    d = so.NDimPropagator()
    d.set_operator(t)
    st.add_propagator(d)
    st.add_transformation(so.FFTTransformation(xg, "k"), so.NORMAL)
    kin = so.kinetic_hamiltonian(xg, 1.0)
    st.add_propagator(so.one_dim_into_propagator(kin, xg, tg, so.FULL))
    p = so.Propagation(so.WaveFunction(a, [lg, xg]), tg, st, precision)
    p.set_timing(True)
    p.steps(1)
    assert "fftpair fx" in " ".join(k[0] for k in p.kernel_times())
    ref = np.fft.ifft(np.fft.fft(a * t, axis=1) * np.exp(-0.01j * kin), axis=1) * t
    got = p.get_array()
    scale = np.abs(ref).max(axis=1, keepdims=True)
    err = np.linalg.norm((got - ref) / scale, axis=1) / np.linalg.norm(ref / scale, axis=1)
    assert err.max() < LANE_TOL[precision], (int(err.argmax()), err.max())
