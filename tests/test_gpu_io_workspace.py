"""Text I/O through the context's kept workspace: texts that grow and shrink,
on changing streams, and values whose text is longer than the room kept per
value (the block of their own).  Exact text."""
import numpy as np
import pytest
import torch

from metada_gb300 import kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("big", [0.0, 0.4, 1.0])
@pytest.mark.parametrize("sizes", [[(1, 1), (700, 300), (7, 5)], [(64, 64), (63, 1), (1, 4097)]])
def test_sizes_streams_and_long_values(dev, sizes, big):
    rng = np.random.default_rng(49)
    streams = [torch.cuda.current_stream(), torch.cuda.Stream(), torch.cuda.Stream()]
    for s, (nx, ny) in zip(streams, sizes):
        v = rng.normal(0.0, 100.0, nx * ny)
        pick = rng.permutation(v.size)[:int(big * min(v.size, 2000))]
        v[pick] = rng.normal(0.0, 1.0, pick.size) * 1e290
        with torch.cuda.stream(s):
            x = torch.from_numpy(v).to(dev)
            text = K.format_state(x, nx, ny)
            back = K.parse_values(text)
        want = "".join(f"{a:12.6f}" + ("\n" if (i + 1) % nx == 0 else " ") for i, a in enumerate(v))
        assert text == want.encode()
        assert np.array_equal(back.cpu().numpy(), np.array([float(t) for t in want.split()]))
