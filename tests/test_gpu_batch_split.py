"""Windows of one call against the same windows one by one: bit for bit wherever no sum depends on how
the call's windows are split over CTAs (the integer Gram matrix of packed frames, in both forms, and no
filter at all)."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,hop,rank", [(32, 8, 2), (64, 16, 4), (128, 32, 4), (64, 64, 0), (50, 25, 0), (48, 16, 3)])
@pytest.mark.parametrize("form", [0, 1])
def test_windows_together_and_alone(cuda, rng, T, hop, rank, form):
    import torch
    import holoflow_b200 as hf
    from holoflow_b200 import pipeline as pl
    H, W, n = 64, 256, 5
    frames = rng.integers(0, 4096, (T + hop * (n - 1)) * H * W).astype(np.uint16)
    dev = torch.from_numpy(O.pack12(frames)).to(cuda)
    cfg = dict(height=H, width=W, frames=T, hop=hop, z_begin=3, z_end=11, clutter_rank=rank, form=form, z=0.27)
    images = []
    for batch in (n, 1):
        p = pl.Pipeline(pl.PipelineConfig(max_batch=batch, **cfg))
        images.append(torch.cat([p.run(dev, T + hop * (n - 1), w * hop, batch) for w in range(0, n, batch)]))
    assert torch.equal(images[0], images[1])
