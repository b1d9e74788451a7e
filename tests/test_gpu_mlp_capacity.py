"""A surrogate handle whose buffers cannot grow (a batch beyond any memory) says
so and stays usable: the batches of before give the results of before, and it
is given back once."""
import ctypes

import pytest
import torch

from metada_gb300 import _lib
from metada_gb300 import kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("call", ["forward", "gradients"])
def test_failed_growth_leaves_the_handle_usable(dev, call):
    mlp = K.MLP(64, 256, 16)
    mlp.init_params(seed=1)
    g = torch.Generator(device=dev)
    g.manual_seed(0)
    X, Y = torch.randn(300, 64, generator=g, device=dev), torch.randn(300, 16, generator=g, device=dev)
    G, loss = mlp.gradients(X, Y)
    out = mlp.forward(X)
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    rows = 1 << 30  # 1 TB an activation: refused before any of the rows is looked at
    if call == "forward":
        rc = mlp.ctx.lib.mg_mlp_forward(mlp.ctx.handle, mlp.handle, p(X), rows, p(out))
    else:
        rc = mlp.ctx.lib.mg_mlp_gradients(mlp.ctx.handle, mlp.handle, p(X), p(Y), rows, p(G), None)
    assert rc == _lib.MG_ERR_NOMEM
    for n in (300, 7):
        G2, loss2 = mlp.gradients(X[:n], Y[:n])
        out2 = mlp.forward(X[:n])
        if n == 300:
            assert torch.equal(G2, G) and abs(loss2 - loss) <= 1e-6 * abs(loss)
        assert torch.equal(out2, out[:n])
    mlp.close()
    torch.cuda.synchronize()
