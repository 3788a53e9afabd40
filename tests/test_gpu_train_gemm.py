"""Training GEMMs at the edges of their tiles.

Gradients of networks whose widths and sample counts are not multiples of the
tiles (odd inputs and outputs take the unaligned copies), against FP64 autograd
of the same network.  Bars: the backward products round both operands to BF16
(relative 2^-9 each), so a layer's weight gradient is within 2^-7 of its norm
plus the rounding of the gradients that reach it (another 2^-7); bias gradients
are FP32 sums of gradients with the same rounding."""
import numpy as np
import pytest

from flint_gb300 import mechgen
from flint_gb300.api import Chemistry
from flint_gb300.surrogate import Surrogate

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("mech,hidden,layers", [("c1", 64, 2), ("c1", 40, 3), ("c2", 256, 3)])
@pytest.mark.parametrize("n", [1, 31, 64, 65, 257, 1000])
def test_gradients(mech, hidden, layers, n):
    chem = Chemistry(mechgen.load(mech))
    ns = chem.ns
    stats = {"x_mean": np.zeros(ns + 2, np.float32), "x_std": np.ones(ns + 2, np.float32),
             "y_mean": np.zeros(ns + 1, np.float32), "y_std": np.ones(ns + 1, np.float32), "bath": ns - 1}
    sur = Surrogate(chem, stats, hidden=hidden, n_layers=layers, seed=3)
    torch.manual_seed(n)
    X = torch.randn(n, ns + 2, device="cuda")
    Yt = torch.randn(n, ns + 1, device="cuda")
    w0, _ = sur.get_state()
    sur.train_step(X, Yt, 1e-3)
    st, _ = sur.get_state()
    g = torch.from_numpy(st[sur.P:2 * sur.P].astype(np.float64)) / 0.1   # first Adam moment = 0.1 gradient
    params, x, o = [], X.double().cpu(), 0
    for l in range(layers):
        a, b = sur.dims[l + 1], sur.dims[l]
        W = torch.from_numpy(w0[o:o + a * b].astype(np.float64)).reshape(a, b).requires_grad_()
        v = torch.from_numpy(w0[o + a * b:o + a * b + a].astype(np.float64)).requires_grad_()
        o += a * b + a
        params += [W, v]
        x = x @ W.t() + v
        if l < layers - 1:
            x = torch.nn.functional.gelu(x, approximate="tanh")
    torch.nn.functional.mse_loss(x, Yt.double().cpu()).backward()
    o = 0
    for p in params:
        got = g[o:o + p.numel()].reshape(p.shape)
        o += p.numel()
        assert (got - p.grad).norm() <= 2.0 ** -6 * p.grad.norm() + 1e-12
