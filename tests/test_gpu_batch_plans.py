"""Plans of the uneven batch beside each other: one of small cases, made after
one of large cases, does not take the large one's kernels their shared memory,
run directly or replayed, in each precision and form."""
import pytest
import torch

from metada_gb300 import _lib
from metada_gb300 import kernels as K

pytestmark = pytest.mark.gpu


def _cases(ks, dev):
    out = []
    for i, k in enumerate(ks):
        g = torch.Generator(device=dev)
        g.manual_seed(7 + i)
        n, p = 700 + i, 130 + i
        rn = lambda *s: torch.randn(s, generator=g, device=dev, dtype=torch.float64)  # noqa: E731
        out.append({"X": rn(k, n) + 3.0, "obs_node": torch.randint(0, n, (p,), generator=g, device=dev),
                    "yo": rn(p) + 3.0, "rvar": torch.ones(p, device=dev, dtype=torch.float64), "rho": 1.1})
    return out


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("precision,flags", [(_lib.MG_PREC_MIXED, 0), (_lib.MG_PREC_MIXED, _lib.MG_COMPAT),
                                             (_lib.MG_PREC_FP64, 0), (_lib.MG_PREC_FP64, _lib.MG_COMPAT)])
def test_small_plan_beside_a_large_one(dev, precision, flags, graph):
    ks = [112, 20, 70]
    dc = _cases(ks, dev)
    X0 = [c["X"].clone() for c in dc]
    large = K.EtkfBatch(dc, flags=flags, precision=precision)
    large.run(graph=False)
    large.finish()
    want = [c["X"].clone() for c in dc]
    small = K.EtkfBatch(_cases([9], dev), flags=flags, precision=precision)
    for c, x in zip(dc, X0):
        c["X"].copy_(x)
    large.run(graph=graph)
    large.finish()
    for c, w in zip(dc, want):
        assert torch.equal(c["X"], w)
    small.run(graph=graph)
    small.finish()


@pytest.mark.parametrize("ks", [[20, 9], [112, 20, 70, 100, 3]])
def test_run_captured_by_the_caller(dev, ks):
    """The chains' streams join the caller's capture and leave it."""
    dc = _cases(ks, dev)
    X0 = [c["X"].clone() for c in dc]
    plan = K.EtkfBatch(dc, flags=0, precision=_lib.MG_PREC_MIXED)
    plan.run(graph=False)
    plan.finish()
    want = [c["X"].clone() for c in dc]
    for c, x in zip(dc, X0):
        c["X"].copy_(x)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        K.context(dev.index)  # the capturing stream
        plan.run(graph=False)
    K.context(dev.index)
    assert all(torch.equal(c["X"], x) for c, x in zip(dc, X0))  # captured, not run
    for _ in range(2):
        for c, x in zip(dc, X0):
            c["X"].copy_(x)
        graph.replay()
        plan.finish()
        assert all(torch.equal(c["X"], w) for c, w in zip(dc, want))
