"""Creating a guess network leaves nothing pending and nothing to be done by its first step."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_weights_set_while_the_default_stream_is_busy():
    """The zeroing of a new network's weights must not run after they are set: the
    network's stream does not wait for the default stream, which is kept busy here."""
    import torch

    from dimspers_b200.learned import GuessNet
    for seed in range(3):
        torch.cuda.synchronize()
        torch.cuda._sleep(200_000_000)     # ~0.1 s on the default stream
        net = GuessNet(9, 16, 8, 3, (1, 2, 1), 2)
        p = np.random.default_rng(seed).standard_normal(net.n).astype(np.float32)
        net.set_params(p)
        torch.cuda.synchronize()
        assert np.array_equal(net.get_params(), p)
        net.close()


def test_the_first_training_step_allocates_nothing():
    import torch

    from dimspers_b200.learned import GuessNet
    x = torch.randn((2, 4, 65, 128), device="cuda")
    t = torch.randn((2, 1, 65, 128), device="cuda")
    free = []
    for _ in range(2):                     # the first network's step also loads the kernels
        net = GuessNet(65, 128, 32, 4, (1, 2, 4, 1), 2)
        net.init_params(0)
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        net.train_step(x, t, 1e-3)
        free.append(before - torch.cuda.mem_get_info()[0])
        net.close()
    assert free[1] == 0
