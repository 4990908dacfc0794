"""A tensor-core product of the network whose bounded wait gave up: the call reports it, and no Adam step
is taken on its result."""
import numpy as np
import pytest

from tests.gpu_common import ensure_built

pytestmark = pytest.mark.gpu


def test_no_step_is_taken_on_a_product_that_gave_up():
    ensure_built()
    import split_operator_gb300 as so
    from split_operator_gb300 import api
    rng = np.random.default_rng(4)
    x = rng.uniform(-1, 1, (100, 5)).astype(np.float32)
    t = rng.standard_normal((100, 7)).astype(np.float32)
    net, other = so.Mlp([5, 32, 7], seed=3), so.Mlp([5, 32, 7], seed=3)
    net.train(x, t, steps=4, lr=1e-2)
    other.train(x, t, steps=4, lr=1e-2)
    before = net.get_params()
    api.selftest_mlp_give_up(net)
    with pytest.raises(Exception, match="gave up"):
        net.train(x, t, steps=300, lr=1e-2)
    np.testing.assert_array_equal(net.get_params(), before)
    for call in (lambda: net.forward(x), lambda: net.gradients(x, t)):
        api.selftest_mlp_give_up(net)
        with pytest.raises(Exception, match="gave up"):
            call()
    # the flag is cleared, and the optimiser goes on from the step it had reached
    net.train(x, t, steps=5, lr=1e-2)
    other.train(x, t, steps=5, lr=1e-2)
    np.testing.assert_array_equal(net.get_params(), other.get_params())


def test_a_batch_without_room_leaves_the_network_usable():
    """The activations of 2^23 rows x 16384 do not fit; what the failed call had already freed is not used
    by the next one."""
    ensure_built()
    import split_operator_gb300 as so
    net = so.Mlp([1, 16384, 1], seed=5)
    x = np.linspace(-1, 1, 10, dtype=np.float32)[:, None]
    first = net.forward(x)
    with pytest.raises(Exception, match="out of memory"):
        net.forward(np.zeros((1 << 23, 1), dtype=np.float32))
    np.testing.assert_array_equal(net.forward(x), first)
    loss, g = net.gradients(x, first)
    assert loss == 0.0 and np.all(np.isfinite(g))
