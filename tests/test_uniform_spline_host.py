"""The basis's own cubic splines against scipy's, and against cubics, which they reproduce."""
import subprocess
import sys

import numpy as np
import pytest

from split_operator_gb300 import learned_start as LS


@pytest.mark.parametrize("n", [4, 5, 17, 1024])
def test_cubics_are_reproduced(n):
    x = np.linspace(-3.0, 5.0, n)
    y = np.stack([np.ones(n), x, x ** 2 - 3.0 * x, 0.5 * x ** 3 - x ** 2 + 1.0], axis=1)
    at = np.concatenate([x, np.linspace(-3.0, 5.0, 301)])
    ref = np.stack([np.ones(len(at)), at, at ** 2 - 3.0 * at, 0.5 * at ** 3 - at ** 2 + 1.0], axis=1)
    # slopes to a few roundings of the largest difference quotient, |y| <= 62
    assert np.abs(LS.uniform_spline(x, y, at) - ref).max() < 1e-12


@pytest.mark.parametrize("n", [2, 3, 5, 64, 1024])
def test_values_match_scipy(n):
    interpolate = pytest.importorskip("scipy.interpolate")
    rng = np.random.default_rng(n)
    x, y = np.linspace(-10.0, 10.0, n), rng.standard_normal((n, 7))
    at = rng.uniform(-10.0, 10.0, 500)
    assert np.abs(LS.uniform_spline(x, y, at) - interpolate.CubicSpline(x, y, axis=0)(at)).max() < 1e-12


def test_a_loaded_basis_predicts_without_scipy():
    """Neither loading the model's module nor summing the basis imports the spline module."""
    code = ("import sys, numpy as np\n"
            "from split_operator_gb300 import learned_start as LS\n"
            "g = LS.Grid2D(nr=64, nth=4)\n"
            "b = LS.RadialBasis(None, None, g, modes=2, nxi=32, u=np.ones((4, 32, 2)))\n"
            "b.state(np.ones((4, 2)), LS.param_sets(1, 0)[0])\n"
            "print('scipy.interpolate' in sys.modules)\n")
    out = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout.strip() == "False", out.stderr
