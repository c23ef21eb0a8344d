"""The tensor-core band passes against the float64 oracle: whole rows (with and without tiles that wait
for a slot of the operand) and row segments (one tile, full segments, a remainder), bin groups that do and
do not fill the epilogue teams, windows of so few rows that a CTA changes window on every unit."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _run(cuda, T, H, W, z0, z1, nwin, dtype, hop):
    import torch
    import holoflow_b200 as hf
    from holoflow_b200 import pipeline as pl
    rng = np.random.default_rng(W + 7 * T + z1)
    n = T + hop * (nwin - 1)
    x = rng.integers(0, 4096, (n, H, W)).astype(np.uint16)
    if dtype == "mono12p":
        ring, dt = torch.from_numpy(O.pack12(x.reshape(-1))).to(cuda), hf.HF_MONO12P
    else:
        ring, dt = torch.from_numpy(x.view(np.int16)).to(cuda), hf.HF_U16
    p = pl.Pipeline(pl.PipelineConfig(height=H, width=W, frames=T, hop=hop, z_begin=z0, z_end=z1, input_dtype=dt, z=0.3,
                                      max_batch=nwin, form=1))
    got = p.run(ring, n, 0, nwin).cpu().numpy()
    assert p.status() == 0
    cfg = O.PathConfig(H, W, T, hop, z0, z1, z=0.3)
    for w in range(nwin):
        exp = O.reconstruct_window(x[w * hop:w * hop + T].astype(np.float64), cfg)
        for m in range(3):  # W to 2^-22, 64..128 float32 sums, two FFT passes: below 1e-4
            assert O.rel_l2(got[w, m], exp[m]) < 1e-4, (w, m)


@pytest.mark.parametrize("dtype", ["mono12p", "u16"])
@pytest.mark.parametrize("W", [256, 512, 768, 1024])
@pytest.mark.parametrize("z0,z1,nwin", [(1, 2, 1), (1, 6, 4), (2, 15, 1), (4, 32, 3), (0, 32, 1)])
def test_band_rows(cuda, dtype, W, z0, z1, nwin):
    _run(cuda, 64, 64, W, z0, z1, nwin, dtype, 16)


@pytest.mark.parametrize("dtype", ["mono12p", "u16"])
@pytest.mark.parametrize("T,W,z0,z1,nwin", [(32, 128, 1, 3, 5), (32, 512, 1, 15, 2), (64, 128, 4, 32, 3), (64, 1536, 1, 9, 1),
                                            (128, 128, 8, 64, 4), (128, 768, 1, 18, 2), (128, 1536, 8, 64, 1)])
def test_band_segments(cuda, dtype, T, W, z0, z1, nwin):
    _run(cuda, T, 64, W, z0, z1, nwin, dtype, 8)
