"""The FP32 band DFT at every light level: dark, mid-range and bright frames, frames of one value, and one
bright frame among dark ones, against float64."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu
TOP = {"u8": 255, "mono12p": 4095, "u16": 65535}


def _frames(rng, fmt, level, T, P):
    top = TOP[fmt]
    if level == "dark":
        return np.minimum(rng.poisson(5, (T, P)), top)
    if level == "bright":
        return np.clip(np.rint(0.9 * top + 0.02 * top * rng.standard_normal((T, P))), 0, top).astype(np.int64)
    if level == "middle":
        return np.clip(np.rint(0.5 * top + 0.1 * top * rng.standard_normal((T, P))), 0, top).astype(np.int64)
    x = np.minimum(rng.poisson(5, (T, P)), top)
    x[{"flash": 0, "late flash": T - 1}[level]] = top
    return x


def _device(x, fmt):
    import torch
    import holoflow_b200 as hf
    if fmt == "mono12p":
        return torch.from_numpy(O.pack12(x.astype(np.uint16).reshape(-1))).cuda(), hf.HF_MONO12P
    if fmt == "u16":
        return torch.from_numpy(x.astype(np.uint16).view(np.int16)).cuda(), hf.HF_U16
    return torch.from_numpy(x.astype(np.uint8)).cuda(), hf.HF_U8


# every unrolled width of the kernel (4 .. 14 bins per thread), one and several groups of bins
@pytest.mark.parametrize("T,z0,z1", [(8, 1, 4), (32, 6, 16), (32, 1, 13), (64, 4, 32), (128, 8, 64)])
@pytest.mark.parametrize("level", ["dark", "middle", "bright", "flash", "late flash"])
@pytest.mark.parametrize("fmt", ["u8", "mono12p", "u16"])
def test_error_follows_the_signal(cuda, rng, fmt, level, T, z0, z1):
    from holoflow_b200 import pipeline as pl
    P = 1026
    x = _frames(rng, fmt, level, T, P)
    dev, dt = _device(x, fmt)
    got = pl.temporal_dft(dev, dt, 1, T, P, z0, z1).cpu().numpy()[0]
    want = np.fft.fft(x.astype(np.float64), axis=0)[z0:z1]
    rms = np.sqrt(np.mean(np.abs(want) ** 2))
    err = np.sqrt(np.mean(np.abs(got - want) ** 2))
    # T float32 roundings of sums as large as a bin's rms (random signs, a few times over), and T rounded
    # roots exp(-2 pi i t k / T) times the pixel's level
    u = 2.0**-24
    assert err <= 8 * u * rms + 2 * u * np.sqrt(T) * x.mean()


@pytest.mark.parametrize("fmt", ["u8", "mono12p", "u16"])
@pytest.mark.parametrize("value", [0, 1, 200])
def test_frames_of_one_value(cuda, fmt, value):
    from holoflow_b200 import pipeline as pl
    T, P = 64, 514
    dev, dt = _device(np.full((T, P), value), fmt)
    got = pl.temporal_dft(dev, dt, 1, T, P, 0, 32).cpu().numpy()[0]
    assert np.array_equal(got[0], np.full(P, T * value, np.complex64))
    assert np.abs(got[1:]).max() <= T * value * 2.0**-24  # the rounded roots' sum
