"""Magnitudes of the column strips and of the row moments with values that leave the range of the
squares: each output is the hypot of its own complex value, whatever stands beside it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _planes(rng, kind, H, W):
    x = (rng.standard_normal((2, H, W)) + 1j * rng.standard_normal((2, H, W))).astype(np.complex64)
    if kind == "zeros":
        x[:] = 0
    elif kind == "impulse":  # magnitudes equal but for the rounding, zeros on the way
        x[:] = 0
        x[:, 0, 0] = 3.0
    elif kind == "infinite":
        x[0, H // 3, W // 2] = np.inf
        x[1, 0, 0] = complex(-np.inf, 1.0)
    elif kind == "nan":
        x[0, 1, 2] = np.nan
    elif kind == "small":
        x *= np.float32(1e-25)
    elif kind == "large":
        x *= np.float32(3e37 / np.sqrt(H * W))
    return x


@pytest.mark.parametrize("H,W", [(64, 64), (256, 64), (512, 256), (768, 64), (1024, 128)])
@pytest.mark.parametrize("kind", ["random", "zeros", "impulse", "infinite", "nan", "small", "large"])
def test_column_magnitudes(cuda, rng, kind, H, W):
    import torch
    import holoflow_b200 as hf
    from holoflow_b200 import pipeline as pl
    x = torch.from_numpy(_planes(rng, kind, H, W)).cuda()
    plans = [pl.FresnelPlan(2, H, W, hf.HF_CF32, 852e-9, 12e-6, 0.3, output_magnitude=m) for m in (False, True)]
    z, mag = (p(x).cpu().numpy() for p in plans)
    with np.errstate(all="ignore"):
        want = np.hypot(z.real, z.imag)
    assert np.array_equal(np.isnan(mag), np.isnan(want))
    assert np.array_equal(np.isinf(mag), np.isinf(want))
    ok = np.isfinite(want)
    assert (np.abs(mag[ok] - want[ok]) <= np.maximum(4 * 2.0**-24 * want[ok], 2.0**-148)).all()
    assert (mag[want == 0] == 0).all()


@pytest.mark.parametrize("side", [256, 1024])
def test_row_moments_of_dark_planes(cuda, side):
    """Angular spectrum of frames of one value: every band plane is zero, and so is every moment."""
    import torch
    import holoflow_b200 as hf
    from holoflow_b200 import pipeline as pl
    T = 32
    cfg = pl.PipelineConfig(side, side, T, T, 6, 16, input_dtype=hf.HF_U8, propagation=hf.HF_PROP_ANGULAR_SPECTRUM)
    p = pl.Pipeline(cfg)
    out = p.run(torch.zeros((T, side, side), dtype=torch.uint8, device="cuda"), T, 0, 1)
    assert torch.count_nonzero(out).item() == 0
