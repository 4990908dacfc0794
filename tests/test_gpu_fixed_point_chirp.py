"""Transform pairs whose length is no power of two: the fixed-point convolutions are no less accurate
than the direct sums in floating point that they stand in for."""
import numpy as np
import pytest

from tests.gpu_common import ensure_built

pytestmark = pytest.mark.gpu


def _pair(a, monkeypatch, fx):
    import split_operator_gb300 as so
    monkeypatch.setenv("SO_FX", fx)
    n = a.shape[-1]
    xg = so.Grid.new_linear_continuos("x", -5.0, 5.0, n, a.ndim - 1)
    grids = [xg] if a.ndim == 1 else [so.Grid.new_linear_countable("lane", 0.0, len(a) - 1.0, len(a), 0), xg]
    tg = so.TimeGrid(0.01, 100)
    st = so.OperationStack()
    st.add_transformation(so.FFTTransformation(xg, "k"), so.NORMAL)
    st.add_propagator(so.one_dim_into_propagator(np.zeros(n), xg, tg, so.FULL))  # factors of one
    p = so.Propagation(so.WaveFunction(a, grids), tg, st, "fp64")
    p.set_timing(True)
    p.steps(1)
    assert (" fx" in " ".join(k[0] for k in p.kernel_times())) == (fx == "1")
    return np.linalg.norm(p.get_array() - a) / np.linalg.norm(a)


# The pair around factors of one gives the state back: what it is off by is the transforms' error.  Two
# convolutions, each rounded at 2^-58 of the lane's bound (at most twice its norm) with the noise of
# four stages, per point: 2^-57 sqrt(2 n) 0.6 is 1.4e-16 to 2.6e-16 for n = 300 to 1000, a third of what the
# sums of n products in FP64 are off by.
@pytest.mark.parametrize("kind", ["packet", "random"])
@pytest.mark.parametrize("n", [18, 100, 300, 500, 514, 1000, 1200, 2050])
def test_pairs_of_other_lengths_are_no_less_accurate(monkeypatch, n, kind):
    ensure_built()
    rng = np.random.default_rng(n)
    if kind == "packet":
        x = np.arange(n) - n // 2
        a = np.stack([np.exp(-(x / (0.03 * n + 1)) ** 2 - 1j * k * x) for k in np.linspace(-1.0, 1.0, 16)])
    else:
        a = rng.standard_normal((16, n)) + 1j * rng.standard_normal((16, n))
    a /= np.linalg.norm(a, axis=1, keepdims=True) * rng.uniform(0.5, 2.0, (16, 1))
    assert _pair(a, monkeypatch, "1") <= _pair(a, monkeypatch, "0")
    if n <= 2048:
        lines = [(_pair(r, monkeypatch, "1"), _pair(r, monkeypatch, "0")) for r in a[::5]]
        assert np.linalg.norm([l[0] for l in lines]) <= np.linalg.norm([l[1] for l in lines])
