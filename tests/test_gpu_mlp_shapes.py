"""Network products at sizes that fill no block: output widths that do not divide by 4, several row
blocks with a ragged last one, and a smaller batch after a larger one on the same network."""
import numpy as np
import pytest

from oracle import mlp_oracle as M
from tests.gpu_common import ensure_built

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def so():
    ensure_built()
    import split_operator_gb300 as so
    return so


def _check(net, widths, batch, seed):
    rng = np.random.default_rng(seed)
    p = net.get_params().astype(np.float64)
    x = rng.uniform(-1, 1, (batch, widths[0])).astype(np.float32)
    t = rng.standard_normal((batch, widths[-1])).astype(np.float32) * 0.3
    loss, g = net.gradients(x, t)
    loss_ref, g_ref = M.loss_and_gradients(p, widths, x, t)
    # the bounds of the gradients' own test: FP32 accumulation against FP64, the same BF16 weights
    assert abs(loss - loss_ref) <= 1e-5 * abs(loss_ref)
    assert np.linalg.norm(g - g_ref) <= 1e-4 * np.linalg.norm(g_ref)
    y, y_ref = net.forward(x), M.forward(p, widths, x)[-1]
    assert np.max(np.abs(y - y_ref)) <= 1e-4 * np.max(np.abs(y_ref))


@pytest.mark.parametrize("widths", [[5, 32, 1], [3, 65, 130, 33], [5, 128, 129, 70], [7, 16, 255]])
def test_ragged_widths_and_batches_match_the_oracle(so, widths):
    net = so.Mlp(widths, seed=2)
    for k, batch in enumerate((1, 129, 300, 127, 128, 5, 257)):
        _check(net, widths, batch, 10 * k + len(widths))
