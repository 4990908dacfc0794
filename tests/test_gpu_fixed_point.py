"""The fixed-point passes of FP64 and float-float states against numpy.

FFT pair [F, K, F^-1, phase]: every power-of-two lane length, tiles that do not divide the lane
count, lanes of very different magnitude, lanes that are zero or not finite.  numpy's FP64
transform pair is within 5e-16 of the exact one (relative L2 per lane), the fixed-point pass
within 4e-16; a float-float result is rounded to 2^-47 per value.  The bounds are twice the sums.
"""
import numpy as np
import pytest

from tests.gpu_common import ensure_built

pytestmark = pytest.mark.gpu

TOL = {"fp64": 2e-15, "float_float": 2e-14}


@pytest.fixture(scope="module")
def so():
    ensure_built()
    import split_operator_gb300 as so
    return so


def _lanes(lanes, n, seed):
    rng = np.random.default_rng(seed)
    x = np.arange(n)
    a = rng.standard_normal((lanes, n)) + 1j * rng.standard_normal((lanes, n))
    # packets, a single point, and magnitudes from 1e-25 to 1e25
    a[1::4] = np.exp(-((x - 0.4 * n) / (0.03 * n + 1.0)) ** 2 + 0.7j * x)
    a[2::4] = 0.0
    a[2::4, n // 3] = 1.0 - 2.0j
    return a * 10.0 ** rng.integers(-25, 26, (lanes, 1))


def _pass(so, a, precision, scale=None):
    """[FFT, kinetic phase, inverse FFT] (scale None), or with a full-size table of magnitude
    `scale` before and after it; an identity matrix along the lane axis keeps the table before the
    transforms in a pass of its own.  Returns (result, reference, the passes' names)."""
    lanes, n = a.shape
    lg = so.Grid.new_linear_countable("lane", 0.0, lanes - 1.0, lanes, 0)
    xg = so.Grid.new_linear_continuos("x", -5.0, 5.0, n, 1)
    tg = so.TimeGrid(0.01, 100)
    st = so.OperationStack()
    t = np.ones((lanes, n), dtype=np.complex128)
    if scale is not None:
        t = scale * np.exp(-1j * np.random.default_rng(n).uniform(-3.0, 3.0, (lanes, n)))
        mt = so.MatrixTransformation(lg, so.Grid.new_linear_countable("same", 0.0, lanes - 1.0, lanes, 0))
        mt.set_diagonalization_matrix(np.eye(lanes), np.eye(lanes))
        st.add_transformation(mt, so.NORMAL)
        ph = so.NDimPropagator()
        ph.set_operator(t)
        st.add_propagator(ph)
    st.add_transformation(so.FFTTransformation(xg, "k"), so.NORMAL)
    kin = so.kinetic_hamiltonian(xg, 1.0)
    st.add_propagator(so.one_dim_into_propagator(kin, xg, tg, so.FULL))
    p = so.Propagation(so.WaveFunction(a, [lg, xg]), tg, st, precision)
    p.set_timing(True)
    p.steps(1)
    with np.errstate(invalid="ignore"):
        ref = np.fft.ifft(np.fft.fft(a * t, axis=1) * np.exp(-0.01j * kin), axis=1) * t
    return p.get_array(), ref, " ".join(k[0] for k in p.kernel_times())


@pytest.mark.parametrize("precision", ["fp64", "float_float"])
@pytest.mark.parametrize("n,lanes", [(16, 600), (32, 37), (64, 5), (128, 700), (256, 37), (512, 2), (1024, 9),
                                     (2048, 37), (4096, 3), (8192, 5)])
def test_fft_pair_lanes_match_numpy(so, precision, n, lanes):
    a = _lanes(lanes, n, 7 * n + lanes)
    got, ref, names = _pass(so, a, precision, 1.0 if lanes <= 37 else None)
    assert "fftpair fx" in names
    err = np.linalg.norm(got - ref, axis=1) / np.linalg.norm(ref, axis=1)
    assert err.max() < TOL[precision], (int(err.argmax()), err.max())


@pytest.mark.parametrize("precision", ["fp64", "float_float"])
@pytest.mark.parametrize("n", [16, 256, 1024, 8192])
def test_lanes_of_zeros_and_of_nan_stay_apart(so, precision, n):
    a = _lanes(6, n, n)
    a[1] = 0.0
    a[3, n // 2] = complex(np.nan, 0.0)
    a[4, 1] = complex(0.0, np.inf)
    got, ref, names = _pass(so, a, precision)
    assert "fftpair fx" in names
    assert np.all(got[1] == 0.0)
    assert np.all(np.isnan(got[3].real)) and np.all(np.isnan(got[4].imag))
    for l in (0, 2, 5):
        assert np.linalg.norm(got[l] - ref[l]) < TOL[precision] * np.linalg.norm(ref[l])


@pytest.mark.parametrize("scale,fixed", [(1.2, True), (0.6, True), (1.3, False), (3.0, False), (0.3, False)])
def test_tables_out_of_the_fixed_point_range_keep_floating_point(so, scale, fixed):
    a = _lanes(4, 1024, 3)
    got, ref, names = _pass(so, a, "fp64", scale)
    assert ("fftpair fx" in names) == fixed
    err = np.linalg.norm(got - ref, axis=1) / np.linalg.norm(ref, axis=1)
    assert err.max() < TOL["fp64"]


@pytest.mark.parametrize("precision", ["fp64", "float_float"])
def test_batch_of_many_short_lanes_equals_single_runs(so, precision):
    """512 points x 256 lanes: the fixed-point pass has more tiles than any pass of the general
    geometry, and the passes recorded before it keep their norm partials."""
    from split_operator_gb300 import workloads as W
    sizes = [(512, 256), (1024, 64), (512, 32)]

    def build():
        return [W.radial_angular_2d(nr=nr, nth=nth, step_no=50, seed=60 + k, r0=52.0, precision=precision)[0]
                for k, (nr, nth) in enumerate(sizes)]

    alone, members = build(), build()
    for p in alone:
        p.steps(6)
    b = so.Batch(members)
    b.steps(6)
    for p, q in zip(alone, members):
        assert np.array_equal(p.get_array(), q.get_array())
        assert p.all_losses() == q.all_losses()
    # the host-to-host call: 4 more steps from the same states
    ins = [p.get_array() for p in members]
    outs = [np.empty_like(a) for a in ins]
    b.steps_host_ptr([a.ctypes.data for a in ins], [a.ctypes.data for a in outs], 4)
    for p, a, o in zip(alone, ins, outs):
        p.set_array(a)
        p.steps(4)
        assert np.array_equal(p.get_array(), o)


# ---- lane matrices on the tensor cores
def _legendre(n):
    x, w = np.polynomial.legendre.leggauss(n)
    v = np.stack([np.sqrt(l + 0.5) * np.polynomial.legendre.Legendre.basis(l)(x) for l in range(n)])
    return v * w[None, :], v.T.copy()


def _matrix_pass(so, a, t, tinv, ph, precision):
    """[T, phase, T^-1] along axis 0: (result, reference in long double, the passes' names)."""
    n, nr = a.shape
    pg = so.Grid.new_linear_countable("p", 0.0, n - 1.0, n, 0)
    rg = so.Grid.new_linear_continuos("r", 0.0, 5.0, nr, 1)
    st = so.OperationStack()
    mt = so.MatrixTransformation(pg, so.Grid.new_linear_countable("l", 0.0, n - 1.0, n, 0))
    mt.set_diagonalization_matrix(t, tinv)
    st.add_transformation(mt, so.NORMAL)
    pd = so.NDimPropagator()
    pd.set_operator(ph)
    st.add_propagator(pd)
    p = so.Propagation(so.WaveFunction(a, [pg, rg]), so.TimeGrid(0.01, 100), st, precision)
    p.set_timing(True)
    p.steps(1)

    def mul(m, z):
        m = m.real.astype(np.longdouble)
        return m @ z.real.astype(np.longdouble) + 1j * (m @ z.imag.astype(np.longdouble))

    with np.errstate(invalid="ignore"):
        ref = mul(tinv, mul(t, a.astype(np.clongdouble)) * ph)
    return p.get_array(), ref, " ".join(k[0] for k in p.kernel_times())


# FP64 sums of n products are within sqrt(n) roundings, the exact sums of 55-bit operands within a
# few: both transforms and the phase stay below 16 roundings (2^-53) of the column; a float-float
# result adds its own 2^-48 per value, grown by the inverse matrix's condition on a column of few l
MAT_TOL = {"fp64": 2e-15, "float_float": 8e-14}


@pytest.mark.parametrize("precision", ["fp64", "float_float"])
@pytest.mark.parametrize("n,nr", [(16, 8), (17, 5), (31, 700), (32, 1216), (33, 64), (64, 7), (100, 2433), (128, 33),
                                  (129, 40), (160, 9), (255, 17), (256, 2448)])
def test_lane_matrices_match_long_double(so, precision, n, nr):
    rng = np.random.default_rng(n + nr)
    t, tinv = _legendre(n)
    a = rng.standard_normal((n, nr)) + 1j * rng.standard_normal((n, nr))
    a[:, 1::3] = tinv[:, :5] @ a[:5, 1::3]           # few l
    a[:, 2::3] = a[:1, 2::3]                          # constant along the lane
    a *= 10.0 ** rng.integers(-25, 25, (1, nr))
    a[:, nr // 2] = 0.0
    a = a.real.astype(np.float32) + 1j * a.imag.astype(np.float32) if precision == "float_float" else a
    ph = np.exp(1j * rng.uniform(0.0, 6.0, (n, nr)))
    got, ref, names = _matrix_pass(so, a.astype(np.complex128), t, tinv, ph, precision)
    assert "tcfx" in names
    assert np.all(got[:, nr // 2] == 0.0)
    live = np.arange(nr) != nr // 2
    err = (np.linalg.norm((got - ref).astype(np.complex128), axis=0)[live] /
           np.linalg.norm(ref.astype(np.complex128), axis=0)[live])
    assert err.max() < MAT_TOL[precision], err.max()


# Every term of a norm is within a few 2^-55 of the largest of its warp's, a partial sum is rounded to
# FP64 once per warp, tile and pass: 2^-50 of the sum of magnitudes holds all of it (float-float:
# the mask is a table of 2^-48)
@pytest.mark.parametrize("precision,tol", [("fp64", 2.0 ** -50), ("float_float", 2.0 ** -45)])
@pytest.mark.parametrize("n,nr", [(16, 8), (33, 4100), (64, 31), (128, 33), (200, 130)])
def test_norms_of_lane_matrix_passes(so, precision, tol, n, nr):
    rng = np.random.default_rng(7 * n + nr)
    t, tinv = _legendre(n)
    # magnitudes from 1e-6 to 1e6 in both axes, weights of either sign and of zero
    a = (rng.standard_normal((n, nr)) + 1j * rng.standard_normal((n, nr))) * 10.0 ** rng.uniform(-6, 6, (1, nr))
    a = (a * 10.0 ** rng.uniform(-6, 6, (n, 1))).astype(np.complex64).astype(np.complex128)
    wp, wr = rng.standard_normal(n), rng.uniform(0.5, 2.0, nr) * 10.0 ** rng.uniform(-3, 3, nr)
    wp[n // 2] = 0.0
    wr[nr // 3] = 0.0
    pg = so.Grid.new_custom("p", np.arange(n, dtype=float), wp, 0)
    rg = so.Grid.new_custom("r", np.arange(nr, dtype=float), wr, 1)
    mask = rng.uniform(0.0, 1.0, nr)
    mask[0] = 1.0
    border = so.BorderDumping(mask.astype(np.complex128), rg)
    border.add_loss_checker("border")
    st = so.OperationStack()
    st.add_control(border, so.FIRST_HALF)
    mt = so.MatrixTransformation(pg, so.Grid.new_linear_countable("l", 0.0, n - 1.0, n, 0))
    mt.set_diagonalization_matrix(t, tinv)
    st.add_transformation(mt, so.NORMAL)
    pd = so.NDimPropagator()
    pd.set_operator(np.exp(1j * rng.uniform(0.0, 6.0, (n, nr))))
    st.add_propagator(pd)
    p = so.Propagation(so.WaveFunction(a, [pg, rg]), so.TimeGrid(0.01, 100), st, precision)
    p.set_timing(True)
    p.steps(1)
    assert "tcfx" in " ".join(k[0] for k in p.kernel_times())
    w = wp.astype(np.longdouble)[:, None] * wr.astype(np.longdouble)[None, :]
    terms = w * (a.real.astype(np.longdouble) ** 2 + a.imag.astype(np.longdouble) ** 2)
    loss = (terms * (1.0 - mask.astype(np.longdouble)[None, :] ** 2)).sum()
    assert abs(p.all_losses()[0] - loss) < tol * np.abs(terms).sum()


# Two masks with loss checkers on both halves: the pass that closes one step and opens the next folds
# five reductions over its tiles.  Two steps of numpy's FP64 and of exact
# digit products differ by some 1e-14 of the norm; split-BF16x6 by 2.2e-7 a step and FP32 sums
# of 16 terms with masks of three roundings (2e-6).
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-13), ("float_float", 1e-12), ("fp32_bf16x6", 5e-6)])
@pytest.mark.parametrize("n,nr", [(128, 4096), (64, 4096)])
def test_many_reductions_in_a_pass(so, precision, tol, n, nr):
    from oracle import split_operator_oracle as O
    rng = np.random.default_rng(n)
    t, tinv = _legendre(n)
    wp = np.polynomial.legendre.leggauss(n)[1]
    wr = rng.uniform(0.5, 2.0, nr)
    a = rng.standard_normal((n, nr)) + 1j * rng.standard_normal((n, nr))
    a /= np.sqrt((np.abs(a) ** 2 * wp[:, None] * wr[None, :]).sum())
    masks = rng.uniform(0.5, 1.0, (2, nr))
    masks[:, 0] = 1.0
    ph = np.exp(1j * rng.uniform(0.0, 6.0, (n, nr)))

    def build(lib):
        pg = lib.Grid.new_custom("p", np.arange(n, dtype=float), wp, 0)
        rg = lib.Grid.new_custom("r", np.arange(nr, dtype=float), wr, 1)
        st = lib.OperationStack()
        for k, m in enumerate(masks):
            b = lib.BorderDumping(m.astype(np.complex128), rg)
            b.add_loss_checker(f"border {k}" if lib is so else lib.LossChecker(f"border {k}"))
            st.add_control(b, lib.FIRST_HALF | lib.SECOND_HALF)
        mt = lib.MatrixTransformation(pg, lib.Grid.new_linear_countable("l", 0.0, n - 1.0, n, 0))
        mt.set_diagonalization_matrix(t, tinv)
        st.add_transformation(mt, lib.NORMAL)
        pd = lib.NDimPropagator()
        pd.set_operator(ph)
        st.add_propagator(pd)
        return lib.WaveFunction(a, [pg, rg]), lib.TimeGrid(0.01, 100), st

    p = so.Propagation(*build(so), precision)
    q = O.Propagation(*build(O))
    p.set_timing(True)
    p.steps(3)
    q.propagate(3)
    assert "tc" in " ".join(k[0] for k in p.kernel_times())
    assert np.abs(np.array(p.all_losses()) - np.array([v for _, v in q.all_losses()])).max() < tol
    assert abs(p.norm() - q.wave_function.norm()) < tol
    assert np.linalg.norm(p.get_array() - q.wave_function.array) < 10 * tol * np.linalg.norm(q.wave_function.array)


@pytest.mark.parametrize("precision", ["fp64", "float_float"])
@pytest.mark.parametrize("nr,nth", [(256, 64), (300, 45)])
def test_plane_steps_do_not_depend_on_the_split(so, precision, nr, nth):
    from split_operator_gb300 import workloads
    whole, _ = workloads.radial_angular_2d(nr=nr, nth=nth, precision=precision)
    whole.steps(6)
    parts, _ = workloads.radial_angular_2d(nr=nr, nth=nth, precision=precision)
    for k in (1, 3, 2):
        parts.steps(k)
    np.testing.assert_array_equal(parts.get_array(), whole.get_array())


def test_columns_that_are_not_finite_stay_apart(so):
    rng = np.random.default_rng(3)
    n, nr = 64, 50
    t, tinv = _legendre(n)
    a = rng.standard_normal((n, nr)) + 1j * rng.standard_normal((n, nr))
    a[5, 7] = complex(np.nan, 1.0)
    a[60, 31] = complex(0.0, np.inf)
    got, ref, names = _matrix_pass(so, a, t, tinv, np.ones((n, nr)), "fp64")
    assert "tcfx" in names
    bad = np.zeros(nr, dtype=bool)
    bad[[7, 31]] = True
    assert np.all(np.isnan(got[:, bad].real))
    err = np.linalg.norm((got - ref).astype(np.complex128)[:, ~bad], axis=0)
    assert np.all(err < MAT_TOL["fp64"] * np.linalg.norm(ref.astype(np.complex128)[:, ~bad], axis=0))


@pytest.mark.parametrize("kind", ["identity", "blocks", "complex", "large_table"])
def test_other_matrices_and_tables_keep_floating_point(so, kind):
    rng = np.random.default_rng(5)
    n, nr = 32, 40
    t, tinv = _legendre(n)
    ph = np.exp(1j * rng.uniform(0.0, 6.0, (n, nr)))
    a = rng.standard_normal((n, nr)) + 1j * rng.standard_normal((n, nr))
    if kind == "identity":
        t = tinv = np.eye(n)
        a[::2] *= 1e-30
    elif kind == "blocks":
        t = np.kron(np.eye(4), rng.standard_normal((8, 8)))
        tinv = t.T.copy()
    elif kind == "complex":
        t = t + 0.1j * t
    else:
        ph = 40.0 * ph
    got, ref, names = _matrix_pass(so, a, t.real if kind != "complex" else t, tinv, ph, "fp64")
    assert "tcfx" not in names
    if kind == "complex":
        ref = ref * (1.0 + 0.1j)
    err = np.abs(got - ref.astype(np.complex128))
    assert np.all(err <= 1e-13 * np.abs(ref).max(axis=1, keepdims=True))


# Lengths that are no power of two: two pairs of inner transforms of M points, each within 4e-16 at
# the filter's two bits of headroom, against numpy's own 1e-15 there
@pytest.mark.parametrize("precision,tol", [("fp64", 4e-15), ("float_float", 2e-14)])
@pytest.mark.parametrize("n,lanes", [(18, 300), (20, 3), (34, 37), (100, 5), (300, 96), (510, 4), (514, 3), (1000, 45),
                                     (2050, 2), (4094, 3)])
def test_fft_pair_of_other_lengths_matches_numpy(so, precision, tol, n, lanes):
    a = _lanes(lanes, n, 11 * n + lanes)
    a[lanes // 2] = 0.0
    got, ref, names = _pass(so, a, precision)
    assert "fftpair fx" in names
    assert np.all(got[lanes // 2] == 0.0)
    live = np.arange(lanes) != lanes // 2
    err = np.linalg.norm(got - ref, axis=1)[live] / np.linalg.norm(ref, axis=1)[live]
    assert err.max() < tol, (int(err.argmax()), err.max())


# ---- resident 1-D propagations
def _line(lib, n, im, x0=0.3, loss=True):
    half = 20.0 * np.sqrt(n / 1024.0)
    grid = lib.Grid.new_linear_continuos("space", -half, half, n, 0)
    x = np.asarray(grid.nodes)
    psi = np.exp(-((x - x0 * half) / 1.7) ** 2 - 0.6j * x)
    wf = lib.WaveFunction(psi.astype(np.complex128), [grid])
    wf.normalize(1.0)
    tg = lib.TimeGrid(0.01, 10 ** 6, im)
    leak = lib.LeakControl()
    if loss:
        leak.add_loss_checker("leak control" if not hasattr(lib, "LossChecker") else lib.LossChecker("leak control"))
    st = lib.OperationStack()
    st.add_control(leak, lib.FIRST_HALF | lib.SECOND_HALF)
    st.add_propagator(lib.one_dim_into_propagator(0.5 * x * x, grid, tg, lib.HALF))
    st.add_transformation(lib.FFTTransformation(grid, "momentum"), lib.NORMAL)
    st.add_propagator(lib.one_dim_into_propagator(lib.kinetic_hamiltonian(grid, 1.0), grid, tg, lib.FULL))
    return wf, tg, st


# 30 steps of numpy's FP64 (5e-16 a step, growing as its square root at best) against as many
# fixed-point steps; the bound is the parity tests' 1e-12 over 30 steps in proportion
# (In imaginary time the packet at x0 decays against the well's centre by e^(-30 dt x0^2 / 2):
# from 2046 points on the rounding noise at the centre, amplified by that, is all that differs.)
@pytest.mark.parametrize("precision,tol", [("fp64", 3e-14), ("float_float", 3e-13)])
@pytest.mark.parametrize("n,im", [(n, False) for n in (16, 18, 32, 34, 64, 100, 128, 256, 500, 512, 1000, 1024, 2046,
                                                       2048, 4096)] +
                         [(n, True) for n in (16, 18, 32, 34, 64, 100, 128, 256, 500, 512, 1000, 1024)])
def test_resident_lines_match_the_oracle(so, precision, tol, n, im):
    from oracle import split_operator_oracle as O
    wf, tg, st = _line(so, n, im)
    owf, otg, ost = _line(O, n, im)
    p = so.Propagation(wf, tg, st, precision)
    q = O.Propagation(owf, otg, ost)
    p.set_timing(True)
    p.steps(30)
    q.propagate(30)
    assert "resident fx" in " ".join(k[0] for k in p.kernel_times())
    a, b = p.get_array(), q.wave_function.array
    assert np.linalg.norm(a - b) < tol * np.linalg.norm(b)
    assert abs(p.norm() - q.wave_function.norm()) < tol
    assert abs(p.all_losses()[0] - q.all_losses()[0][1]) < 30 * tol


@pytest.mark.parametrize("n", [256, 500, 2048])
def test_resident_lines_do_not_depend_on_the_split(so, n):
    wf, tg, st = _line(so, n, True)
    whole = so.Propagation(wf, tg, st, "fp64")
    whole.steps(23)
    wf2, tg2, st2 = _line(so, n, True)
    parts = so.Propagation(wf2, tg2, st2, "fp64")
    for k in (1, 7, 2, 13):
        parts.steps(k)
    np.testing.assert_array_equal(parts.get_array(), whole.get_array())
    assert parts.all_losses() == whole.all_losses()
    assert parts.norm() == whole.norm()


@pytest.mark.parametrize("n", [64, 500])
def test_resident_line_with_nan_or_zero(so, n):
    wf, tg, st = _line(so, n, False)
    p = so.Propagation(wf, tg, st, "fp64")
    a = p.get_array()
    a[3] = complex(np.nan, 0.0)
    p.set_array(a)
    p.steps(3)
    assert np.all(np.isnan(p.get_array().real))
    from split_operator_gb300._lib import SplitOperatorError
    with pytest.raises(SplitOperatorError):
        p.synchronize()
