"""Weight gradients summed over a split batch: sizes at the edges of the
tiles (64 x 64, 16-wide for narrow sides), of the K steps (16 rows) and of
the split, aligned and not, against the numpy oracle."""
import numpy as np
import pytest
import torch

from conftest import rel_err

import oracle.mlp as om
from metada_gb300 import kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,nin,nh,nout", [(1, 6, 10, 3), (63, 13, 70, 17), (64, 64, 64, 16), (129, 16, 65, 32),
                                           (1000, 60, 256, 16), (4099, 64, 96, 1), (16385, 5, 130, 31)])
def test_split_gradients(dev, B, nin, nh, nout):
    mlp = K.MLP(nin, nh, nout)
    mlp.init_params(seed=B)
    g = np.random.default_rng(B)
    X = g.standard_normal((B, nin)).astype(np.float32)
    Yt = g.standard_normal((B, nout)).astype(np.float32)
    G, loss = mlp.gradients(torch.tensor(X, device=dev), torch.tensor(Yt, device=dev))
    Pw = mlp.params(bf16_rounded=True).cpu().numpy().astype(np.float64)  # init biases are zero
    want, wloss = om.gradients(Pw, X, Yt, np.zeros(nout, np.float32), np.ones(nout, np.float32), nin, nh, nout)
    got, want = G.cpu().numpy(), np.asarray(want)
    for part in om.unpack(np.arange(mlp.nparam), nin, nh, nout):  # each weight and bias block on its own scale
        i = part.reshape(-1).astype(int)
        assert rel_err(got[i], want[i]) <= 1e-4
    assert abs(loss - wloss) <= 1e-4 * wloss
