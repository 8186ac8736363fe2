"""The gradient of a large batch of equal elements is one element's (the loss is a mean): a sum over
elements that loses digits as it grows shows.  All terms of a sum have one sign, so its relative
error is at most the length of its longest chain of FP32 additions times 2^-24: 512 nodes, the
elements of a CTA (at most 400 here), 8 runs of 19 CTAs, and twice 432 for the activations that
enter: 1803 * 2^-24 = 1.1e-4."""
import numpy as np
import pytest
import torch

from test_net_train_gpu import conv, gelu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Nq,C,E", [(8, 16, 60800), (8, 4, 240000), (6, 16, 120000), (4, 8, 200000)])
def test_gradient_of_equal_elements(nb, dev, Nq, C, E):
    rng = np.random.default_rng(Nq + C)
    net = nb.Net(Nq, C, 3, seed=2)
    w = rng.uniform(0.01, 0.05, net.weights().size).astype(np.float32)
    net.set_weights(w)
    x = rng.uniform(0.5, 1.5, (1, 1, Nq, Nq, Nq)).astype(np.float32)
    y = -rng.uniform(0.5, 1.5, (1, 1, Nq, Nq, Nq)).astype(np.float32)
    all_of = lambda a: torch.from_numpy(a).to(dev).expand(E, -1, -1, -1, -1).contiguous()  # noqa: E731
    g, loss = net.gradient(all_of(x), all_of(y), E)
    W = torch.from_numpy(w.astype(np.float64)).requires_grad_()
    w1, w2, w3 = torch.split(W, (27 * C, 27 * C * C, 27 * C))
    h = gelu(conv(torch.from_numpy(x).double(), w1.view(C, 1, 3, 3, 3)))
    h = gelu(conv(h, w2.view(C, C, 3, 3, 3)))
    ref = ((conv(h, w3.view(1, C, 3, 3, 3)) - torch.from_numpy(y).double()) ** 2).mean()
    ref.backward()
    r = W.grad.numpy()
    assert abs(loss - float(ref.detach())) <= 1.1e-4 * float(ref.detach())
    assert np.all(abs(g - r) <= 1.1e-4 * abs(r))
