"""Input statistics of a guess network as a program may set them: in 64 bits (applied in
64 bits, one rounding to FP32 each, as torch does it in place), and four of them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def setup(ctx, dtype):
    from dimspers_b200.learned import GuessNet, grid_shape
    net = GuessNet(*grid_shape(16, 64), 8, 3, (1, 2, 1), 1)
    net.init_params(2)
    net.x_mean = np.array([0.1, -0.3, 0.7, 1 / 3]).astype(dtype)
    net.x_std = np.array([1.1, 0.7, 1 / 3, 0.9]).astype(dtype)
    net.y_mean, net.y_std = 0.3, 1.7
    return net


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_statistics_are_applied_in_their_own_precision(dtype):
    import torch

    from dimspers_b200 import StokesContext, inputs
    from dimspers_b200.learned import LearnedGuess, features
    with StokesContext(16, 64, "discontinuous") as c:
        m = inputs.make_material(c.mesh, "aniso", seed=3)
        c.set_material_ti(m.eta_ip, m.rho, m.g, m.delta, m.dir_x, m.dir_y)
        net = setup(c, dtype)
        guess = LearnedGuess(net, c)
        P = torch.empty(c.npres, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        guess.predict(m.g, P.data_ptr())
        x = torch.empty_like(guess.x)
        torch.cuda.synchronize()
        features(c, x)
        x = x.cpu()
        for v, op in ((net.x_mean, x.sub_), (net.x_std, x.div_)):
            op(torch.from_numpy(v).view(1, 4, 1, 1))
        assert torch.equal(guess.x.cpu(), x)
        xd, y = x.cuda(), torch.empty_like(guess.y)
        torch.cuda.synchronize()
        net.forward(xd, y)
        y = y.cpu().mul_(net.y_std).add_(net.y_mean)
        assert torch.equal(guess.y.cpu(), y)
        assert bool(torch.isfinite(P).all())
        net.close()


def test_statistics_of_another_length_are_refused():
    from dimspers_b200 import StokesContext
    from dimspers_b200.learned import LearnedGuess
    with StokesContext(16, 64, "discontinuous") as c:
        net = setup(c, np.float32)
        net.x_mean = net.x_mean[:3]
        with pytest.raises(Exception):
            LearnedGuess(net, c)
        net.close()
