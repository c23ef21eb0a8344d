"""Gram matrices of the frames that are summed in float64 (T other than 32, 64, 128, P % 8 != 0, rows or a
base that are not 4-byte aligned): exact for integer samples, float64 rounding for float frames, by every
entry point, and by hf_covariance_noalloc without shared state."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _device(x, fmt, lead=0):
    """Samples [B][T][P] on the device, `lead` bytes after an aligned address."""
    import torch
    import holoflow_b200 as hf
    host, dt = {"mono12p": (lambda: O.pack12(x.astype(np.uint16).reshape(-1)), hf.HF_MONO12P),
                "u16": (lambda: x.astype(np.uint16), hf.HF_U16), "u8": (lambda: x.astype(np.uint8), hf.HF_U8),
                "f32": (lambda: x.astype(np.float32), hf.HF_F32)}[fmt]
    raw = np.ascontiguousarray(host()).reshape(-1).view(np.uint8)
    buf = torch.zeros(raw.size + lead, dtype=torch.uint8, device="cuda")
    buf[lead:] = torch.from_numpy(raw).cuda()
    return buf[lead:], dt


def _samples(rng, fmt, shape):
    if fmt == "f32":  # a strong constant part
        return (3000.0 + 50.0 * rng.standard_normal(shape)).astype(np.float32).astype(np.float64)
    return rng.integers(0, {"u8": 256, "u16": 65536, "mono12p": 4096}[fmt], shape).astype(np.float64)


def _check(got, x, fmt):
    for b in range(x.shape[0]):
        G = x[b] @ x[b].T
        if fmt == "f32":  # P additions of 2^-53 each, here and in numpy
            assert np.abs(got[b] - G).max() <= 2 * x.shape[2] * 2.0**-53 * np.abs(G).max()
        else:
            assert np.array_equal(got[b], G)


# one and several 8-frame blocks, remainders of blocks and tiles, one CTA per window (300 windows), many
# tiles per CTA, and rows, sides or bases that exclude the FP32 sums at T = 32, 64, 128
@pytest.mark.parametrize("fmt,B,T,P,lead", [
    ("u16", 1, 1, 5, 0), ("u16", 2, 3, 1000, 0), ("u8", 2, 16, 333, 0), ("mono12p", 2, 17, 4098, 0),
    ("u16", 300, 50, 700, 0), ("u16", 1, 50, 300001, 0), ("f32", 2, 50, 20000, 0), ("f32", 300, 9, 257, 0),
    ("u8", 2, 100, 5000, 0), ("f32", 1, 127, 3001, 0), ("mono12p", 1, 127, 3002, 0), ("u16", 2, 32, 4099, 0),
    ("u16", 2, 64, 4096, 2), ("u8", 2, 64, 4096, 3), ("mono12p", 2, 128, 2048, 1), ("f32", 2, 128, 1001, 0),
    ("u16", 2, 130, 600, 0), ("f32", 1, 200, 777, 0), ("u8", 64, 8, 1024, 0), ("mono12p", 3, 24, 254, 0)])
def test_float64_sums(cuda, rng, fmt, B, T, P, lead):
    from holoflow_b200 import pipeline as pl
    import torch
    x = _samples(rng, fmt, (B, T, P))
    dev, dt = _device(x, fmt, lead)
    _check(pl.covariance(dev, dt, B, T, P).cpu().numpy(), x, fmt)
    if P <= 5000:
        g = torch.empty((B, T, T), dtype=torch.float64, device="cuda")
        _check(pl.covariance_noalloc(dev, dt, B, T, P, g).cpu().numpy(), x, fmt)


def test_plan_of_other_sizes_is_exact(cuda, rng):
    import torch
    import holoflow_b200 as hf
    from holoflow_b200 import pipeline as pl
    H, W, T, hop = 75, 101, 50, 25
    x = rng.integers(0, 65536, (T + hop, H * W))
    cfg = pl.PipelineConfig(H, W, T, hop, 2, 6, input_dtype=hf.HF_U16, clutter_rank=2, max_batch=2)
    p = pl.Pipeline(cfg)
    p.run(torch.from_numpy(x.astype(np.uint16).view(np.int16)).cuda(), T + hop, 0, 2)
    for w in range(2):
        X = x[w * hop:w * hop + T].astype(np.float64)
        assert np.array_equal(p.inspect(w)[0].cpu().numpy(), X @ X.T)


def test_noalloc_calls_without_workspace_overlap(cuda, rng):
    """Two streams at once: shapes that are summed in float64 use nothing in common."""
    import torch
    from holoflow_b200 import pipeline as pl
    streams, jobs = [torch.cuda.Stream() for _ in range(2)], []
    for s in streams:
        x = _samples(rng, "u16", (8, 40, 3000))
        dev, dt = _device(x, "u16")
        jobs.append((s, x, dev, dt, torch.empty((8, 40, 40), dtype=torch.float64, device="cuda")))
    torch.cuda.synchronize()
    for _ in range(10):
        for s, x, dev, dt, g in jobs:
            with torch.cuda.stream(s):
                pl.covariance_noalloc(dev, dt, 8, 40, 3000, g)
    torch.cuda.synchronize()
    for s, x, dev, dt, g in jobs:
        _check(g.cpu().numpy(), x, "u16")


# Many windows with few partials, few with many, and the batches on either side of a full wave of CTAs.
# Samples within 8 of the shift: every FP32 sum is a small integer, so the matrix is exact however it is
# split and reduced.
@pytest.mark.parametrize("fmt,B,T,P", [("u16", 64, 128, 1024), ("u16", 16, 64, 16384), ("u8", 7, 128, 1024), ("u16", 9, 32, 8192),
                                       ("f32", 296, 32, 512), ("u16", 297, 32, 64), ("mono12p", 1, 128, 65536)])
def test_split_and_reduction_of_fp32_sums(cuda, rng, fmt, B, T, P):
    from holoflow_b200 import pipeline as pl
    x = rng.integers(-8, 9, (B, T, P)).astype(np.float64) + {"u8": 128, "u16": 2048, "mono12p": 2048, "f32": 0}[fmt]
    dev, dt = _device(x, fmt)
    got = pl.covariance(dev, dt, B, T, P).cpu().numpy()
    for b in range(B):
        assert np.array_equal(got[b], x[b] @ x[b].T)
