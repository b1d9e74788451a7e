"""A training step captured after a forward pass of the same size: nothing is
left to allocate, and the replayed step is the step."""
import pytest
import torch

from metada_gb300 import kernels as K

pytestmark = pytest.mark.gpu


def test_training_step_captured_after_a_forward_pass(dev):
    g = torch.Generator(device=dev)
    g.manual_seed(3)
    X, Y = torch.randn(500, 64, generator=g, device=dev), torch.randn(500, 16, generator=g, device=dev)
    steps = []
    for captured in (False, True):
        mlp = K.MLP(64, 256, 16)
        P0 = mlp.init_params(seed=5)
        mlp.forward(X)
        torch.cuda.synchronize()
        if captured:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                K.context(dev.index)  # the capturing stream
                mlp.train_step(X, Y, 1e-3)
            K.context(dev.index)
            assert torch.equal(mlp.params(), P0)  # captured, not run
            graph.replay()
        else:
            mlp.train_step(X, Y, 1e-3)
        torch.cuda.synchronize()
        steps.append(mlp.params() - P0)
    assert steps[0].abs().max() > 0 and torch.equal(steps[0], steps[1])
