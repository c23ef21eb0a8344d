"""The ring-fed row passes at the row counts where their launch changes: fewer rows than SMs, one warp
more per CTA, one round more, against the float64 oracle."""
import math

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


# rows / 148 SMs: one warp per CTA, two, up to the most warps of the length and a round more
@pytest.mark.parametrize("rows,W", [(1, 64), (147, 64), (148, 128), (149, 64), (593, 256), (2368, 64), (2369, 128),
                                    (4737, 64), (512, 512), (1776, 768), (1777, 768), (2304, 768), (1184, 1536),
                                    (1185, 1536), (5, 1024), (1780, 1024)])
def test_row_counts(cuda, rows, W):
    import torch
    import holoflow_b200 as hf
    from holoflow_b200 import pipeline as pl
    rng = np.random.default_rng(rows + W)
    x = (rng.standard_normal((rows, 1, W)) + 1j * rng.standard_normal((rows, 1, W))).astype(np.complex64)
    plan = pl.FresnelPlan(rows, 1, W, hf.HF_CF32, 852e-9, 12e-6, 0.2)
    exp = O.fresnel(x, 852e-9, 12e-6, 12e-6, 0.2)
    assert O.rel_l2(plan(torch.from_numpy(x).cuda()).cpu().numpy(), exp) < 2e-6 * math.log2(W)  # as the other Fresnel tests


@pytest.mark.parametrize("H,W,nwin", [(64, 64, 1), (256, 64, 1), (256, 64, 4), (768, 128, 1), (512, 256, 3), (1024, 64, 2)])
def test_moment_row_counts(cuda, H, W, nwin):
    import torch
    import holoflow_b200 as hf
    from holoflow_b200 import pipeline as pl
    rng = np.random.default_rng(H)
    T, z0, z1 = 16, 2, 7
    frames = rng.integers(0, 4096, (T * nwin, H, W)).astype(np.uint16)
    cfg = dict(z=0.27, fs=37e3, propagation="angular_spectrum")
    p = pl.Pipeline(pl.PipelineConfig(H, W, T, T, z0, z1, input_dtype=hf.HF_U16, propagation=hf.HF_PROP_ANGULAR_SPECTRUM,
                                      max_batch=nwin, z=0.27, fs=37e3))
    out = p.run(torch.from_numpy(frames.view(np.int16)).cuda(), T * nwin, 0, nwin).cpu().numpy()
    for w in range(nwin):
        exp = O.reconstruct_window(frames[w * T:(w + 1) * T], O.PathConfig(H, W, T, T, z0, z1, **cfg))
        for m in range(3):
            assert O.rel_l2(out[w, m], exp[m]) < 1e-4  # the plain form's tolerance
