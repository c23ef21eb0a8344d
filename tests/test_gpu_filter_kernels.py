"""The clutter filter's kernels at the edges of their dispatch: the exact integer Gram matrix (window
lengths, hops on and off the 8-frame grid, partial pixel tiles, both forms), the top-r eigensolver on
matrices at scratch limits, and the filter matrix with and without its staged tables."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [32, 64, 128])
@pytest.mark.parametrize("fmt", ["mono12p", "u8"])
@pytest.mark.parametrize("hop,nwin,H,W", [(8, 5, 4, 40), (16, 3, 8, 100), (24, 2, 32, 36), (32, 9, 16, 64),
                                          (5, 3, 4, 8), (64, 2, 64, 64), (16, 1, 96, 128)])
@pytest.mark.parametrize("form", [0, 1])
def test_integer_gram_is_exact(cuda, T, fmt, hop, nwin, H, W, form):
    import torch
    import holoflow_b200 as hf
    from holoflow_b200 import pipeline as pl
    rng = np.random.default_rng(T + hop)
    n = T + hop * (nwin - 1) + 3
    x = rng.integers(0, 4096 if fmt == "mono12p" else 256, (n, H, W))
    x[0], x[1] = 0, 4095 if fmt == "mono12p" else 255  # both ends of the sample range
    if fmt == "mono12p":
        ring, dt = torch.from_numpy(O.pack12(x.astype(np.uint16).reshape(-1))).to(cuda), hf.HF_MONO12P
    else:
        ring, dt = torch.from_numpy(x.astype(np.uint8)).to(cuda), hf.HF_U8
    p = pl.Pipeline(pl.PipelineConfig(height=H, width=W, frames=T, hop=hop, z_begin=1, z_end=4, input_dtype=dt,
                                      propagation=hf.HF_PROP_NONE, clutter_rank=1, max_batch=nwin, form=form))
    first = 2
    p.run(ring, n, first, nwin)
    for w in range(nwin):
        gram, _ = p.inspect(w)
        f = x[[(first + w * hop + t) % n for t in range(T)]].reshape(T, -1).astype(np.int64)
        assert np.array_equal(gram.cpu().numpy(), (f @ f.T).astype(np.float64)), w
    assert p.status() == 0
