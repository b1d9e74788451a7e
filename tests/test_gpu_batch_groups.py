"""The mixed uneven batch runs its cases in up to three chains on streams of
their own.  A case's analysis does not depend on the others: with one, two or
three groups present, run directly (twice, on changing streams) or replayed
from the graph, every case's members are bit-identical to the case alone."""
import numpy as np
import pytest
import torch

from metada_gb300 import _lib
from metada_gb300 import kernels as K

pytestmark = pytest.mark.gpu


def _cases(ks, dev):
    out = []
    for i, k in enumerate(ks):
        g = np.random.default_rng(100 + i)
        n, p = int(g.integers(300, 3000)), int(g.integers(1, 1500))
        X = 280.0 + g.normal(0, 1, (k, n))
        out.append({"X": torch.tensor(X, device=dev), "obs_node": torch.tensor(g.integers(0, n, p), device=dev),
                    "yo": torch.tensor(280.0 + g.normal(0, 1, p), device=dev),
                    "rvar": torch.full((p,), 0.5, dtype=torch.float64, device=dev), "rho": 1.1})
    return out


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("ks", [[112], [64, 2], [65, 112, 80], [112, 32], [3, 33, 64, 65, 88, 96, 111, 112, 100, 17]])
def test_groups_bit_identical_to_single_cases(dev, ks, graph):
    dc = _cases(ks, dev)
    X0 = [c["X"].clone() for c in dc]
    want = []
    for c, x in zip(dc, X0):
        one = dict(c, X=x.clone())
        b = K.EtkfBatch([one], flags=0, precision=_lib.MG_PREC_MIXED)
        b.run(graph=False)
        b.finish()
        want.append(one["X"])
    b = K.EtkfBatch(dc, flags=0, precision=_lib.MG_PREC_MIXED)
    for stream in (torch.cuda.current_stream(), torch.cuda.Stream()):
        with torch.cuda.stream(stream):
            for c, x in zip(dc, X0):
                c["X"].copy_(x)
            b.run(graph=graph)
            ms = b.finish()
        assert np.all(np.asarray(ms) > 0)
        for c, w in zip(dc, want):
            assert torch.equal(c["X"], w)
