"""The FP32 band DFT at the edges of its dispatch: every bin-group size, partial tiles, rows aligned to
16, 4 and fewer bytes, 16- and 8-byte stores, and each sample format."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _frames(rng, fmt, shape):
    top = {"u8": 256, "f32": 4096, "u16": 65536, "mono12p": 4096}[fmt]
    return rng.integers(0, top, shape)


def _device(cuda, x, fmt, offset=0):
    import torch
    if fmt == "mono12p":
        raw = O.pack12(x.astype(np.uint16).reshape(-1))
    elif fmt == "u16":
        raw = x.astype(np.uint16).reshape(-1).view(np.uint8)
    elif fmt == "u8":
        raw = x.astype(np.uint8).reshape(-1)
    else:
        raw = x.astype(np.float32).reshape(-1).view(np.uint8)
    buf = torch.zeros(raw.size + offset, dtype=torch.uint8, device=cuda)
    buf[offset:] = torch.from_numpy(raw.copy()).to(cuda)
    return buf[offset:]


# tolerance: FP32 sums of T products against float64, as the other temporal-DFT tests
@pytest.mark.parametrize("fmt", ["u8", "u16", "mono12p", "f32"])
@pytest.mark.parametrize("T,P,z0,z1", [(64, 1024, 4, 32), (32, 514, 0, 17), (16, 2050, 1, 2), (7, 126, 0, 7),
                                       (128, 1000, 8, 64), (50, 390, 3, 15), (64, 128, 0, 33), (33, 4100, 1, 7),
                                       (128, 384, 0, 65), (3, 6, 0, 3), (200, 130, 0, 100)])
def test_band_dft_shapes(cuda, fmt, T, P, z0, z1):
    import holoflow_b200 as hf
    from holoflow_b200 import pipeline as pl
    rng = np.random.default_rng(T * P)
    dt = {"u8": hf.HF_U8, "u16": hf.HF_U16, "mono12p": hf.HF_MONO12P, "f32": hf.HF_F32}[fmt]
    x = _frames(rng, fmt, (2, T, P))
    got = pl.temporal_dft(_device(cuda, x, fmt), dt, 2, T, P, z0, z1).cpu().numpy()
    assert O.rel_l2(got, np.fft.fft(x, axis=1)[:, z0:z1]) < 1e-5


@pytest.mark.parametrize("fmt,offset,P", [("u8", 1, 1025), ("u8", 4, 1028), ("u8", 16, 999), ("u16", 2, 1023),
                                          ("u16", 4, 514), ("f32", 4, 777), ("mono12p", 1, 1026),
                                          ("mono12p", 4, 1032)])
def test_band_dft_alignments(cuda, fmt, offset, P):
    import torch
    import holoflow_b200 as hf
    from holoflow_b200 import pipeline as pl
    rng = np.random.default_rng(P)
    T, z0, z1 = 32, 2, 13
    dt = {"u8": hf.HF_U8, "u16": hf.HF_U16, "mono12p": hf.HF_MONO12P, "f32": hf.HF_F32}[fmt]
    x = _frames(rng, fmt, (2, T, P))
    dev = _device(cuda, x, fmt, offset)
    exp = np.fft.fft(x, axis=1)[:, z0:z1]
    n = 2 * (z1 - z0) * P
    for shift in (0, 1):  # the output 16-byte aligned, then only 8-byte aligned
        out = torch.zeros(n + 2, dtype=torch.complex64, device=cuda)
        hf.check(hf.lib().hf_temporal_dft(pl._ptr(dev), dt, 2, T, P, z0, z1, 0, pl._ptr(out[shift:]), pl._stream()))
        o = out.cpu().numpy()
        assert O.rel_l2(o[shift:shift + n].reshape(exp.shape), exp) < 1e-5
        assert not o[:shift].any() and not o[shift + n:].any()  # nothing outside the planes
