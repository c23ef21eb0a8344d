"""The ring-fed row passes and the transfer-function columns: every four-step length, row counts that
do not fill the warps, placement in a padded plane (its empty rows skipped), both directions, and
inputs the ring does not take (odd margins, 8-byte-aligned bases) against the float64 oracle."""
import math

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

LAM, DX = 852e-9, 12e-6


def _complex(rng, shape):
    return (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)


@pytest.mark.parametrize("W", [64, 128, 256, 512, 768, 1024, 1536])
@pytest.mark.parametrize("H", [1, 7, 64])
def test_fresnel_row_lengths(cuda, H, W):
    import torch
    import holoflow_b200 as hf
    from holoflow_b200 import pipeline as pl
    rng = np.random.default_rng(W + H)
    x = _complex(rng, (3, H, W))
    plan = pl.FresnelPlan(3, H, W, hf.HF_CF32, LAM, DX, 0.2)
    exp = O.fresnel(x, LAM, DX, DX, 0.2)
    tol = 2e-6 * math.log2(H * W)  # the bound of the other Fresnel tests
    buf = torch.zeros(x.size + 1, dtype=torch.complex64, device=cuda)
    for off in (0, 1):  # 16-byte aligned, then only 8-byte aligned
        v = buf[off:off + x.size].view(3, H, W)
        v.copy_(torch.from_numpy(x))
        assert O.rel_l2(plan(v).cpu().numpy(), exp) < tol


@pytest.mark.parametrize("B,H,W,pad,real,inplace", [
    (2, 64, 64, None, False, True), (3, 128, 256, None, False, False), (1, 256, 1536, None, False, True),
    (2, 60, 100, (128, 64), False, False), (2, 60, 100, (128, 64), True, False), (1, 62, 254, (256, 64), False, False),
    (1, 126, 510, (512, 256), False, False), (1, 700, 768, (768, 768), False, False),
    (1, 1024, 1022, (1024, 1024), False, False), (5, 512, 512, None, False, True)])
def test_angular_spectrum_four_step(cuda, B, H, W, pad, real, inplace):
    import torch
    import holoflow_b200 as hf
    from holoflow_b200 import pipeline as pl
    rng = np.random.default_rng(W)
    x = rng.standard_normal((B, H, W)).astype(np.float32) if real else _complex(rng, (B, H, W))
    padding = {"width": pad[0], "height": pad[1]} if pad else None
    filt = {"r_inner": 3, "r_outer": 25, "s_inner": 2, "s_outer": 6}
    plan = pl.AngularSpectrumPlan(B, H, W, hf.HF_F32 if real else hf.HF_CF32, LAM, DX, 0.3, padding, filt)
    exp = O.angular_spectrum(x, LAM, DX, DX, 0.3, filt, padding)
    n = exp.size
    for off in (0, 1):  # output 16-byte aligned, then only 8-byte aligned (the older kernels)
        dev = torch.from_numpy(x).to(cuda)
        buf = torch.full((n + 2,), float("nan"), dtype=torch.complex64, device=cuda)
        out = buf[off:off + n].view(*exp.shape)
        if inplace:
            out.copy_(dev)
            dev = out
        got = plan(dev, out).cpu().numpy()
        assert O.rel_l2(got, exp) < 5e-5, off  # the bound of the other angular-spectrum tests


@pytest.mark.parametrize("H,W,pad,nwin,dtype", [(64, 64, None, 3, "u16"), (128, 512, None, 1, "mono12p"),
                                                (100, 200, (256, 128), 2, "u8"), (256, 768, None, 2, "u16"),
                                                (50, 1000, (1024, 64), 1, "u16"), (64, 1536, None, 1, "mono12p")])
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("mask", [7, 5])
def test_angular_moments(cuda, H, W, pad, nwin, dtype, shift, mask):
    import torch
    import holoflow_b200 as hf
    from holoflow_b200 import pipeline as pl
    rng = np.random.default_rng(H * W)
    T, z0, z1 = 16, 1, 6
    x = rng.integers(0, 256 if dtype == "u8" else 4096, (T * nwin, H, W)).astype(np.uint16)
    if dtype == "mono12p":
        ring, dt = torch.from_numpy(O.pack12(x.reshape(-1))).to(cuda), hf.HF_MONO12P
    elif dtype == "u8":
        ring, dt = torch.from_numpy(x.astype(np.uint8)).to(cuda), hf.HF_U8
    else:
        ring, dt = torch.from_numpy(x.view(np.int16)).to(cuda), hf.HF_U16
    pw, ph = pad if pad else (0, 0)
    p = pl.Pipeline(pl.PipelineConfig(height=H, width=W, frames=T, hop=T, z_begin=z0, z_end=z1, input_dtype=dt, z=0.3,
                                      propagation=hf.HF_PROP_ANGULAR_SPECTRUM, max_batch=nwin, pad_w=pw, pad_h=ph,
                                      fftshift=shift, moment_mask=mask))
    got = p.run(ring, T * nwin, 0, nwin).cpu().numpy()
    cfg = O.PathConfig(H, W, T, T, z0, z1, z=0.3, propagation="angular_spectrum", fftshift=bool(shift),
                       as_padding={"width": pw, "height": ph} if pad else None)
    for w in range(nwin):
        exp = O.reconstruct_window(x[w * T:(w + 1) * T].astype(np.float64), cfg)
        for i, m in enumerate([m for m in range(3) if mask >> m & 1]):
            assert O.rel_l2(got[w, i], exp[m]) < 1e-4, (w, m)


@pytest.mark.parametrize("H,W,nwin", [(64, 64, 1), (64, 256, 3), (128, 64, 2), (128, 1024, 1), (256, 128, 1), (256, 512, 2),
                                      (512, 64, 1), (512, 768, 1)])
@pytest.mark.parametrize("nz", [1, 4, 5, 16, 31])
@pytest.mark.parametrize("shift,mask,form", [(0, 7, 0), (1, 6, 1)])
def test_short_column_moments(cuda, H, W, nwin, nz, shift, mask, form):
    """Groups of planes in the column pass: one plane, full groups, a remainder, both CTA sizes."""
    import torch
    import holoflow_b200 as hf
    from holoflow_b200 import pipeline as pl
    rng = np.random.default_rng(H * W + nz)
    T, z0 = 64, 1
    x = rng.integers(0, 4096, (T * nwin, H, W)).astype(np.uint16)
    ring = torch.from_numpy(x.view(np.int16)).to(cuda)
    p = pl.Pipeline(pl.PipelineConfig(height=H, width=W, frames=T, hop=T, z_begin=z0, z_end=z0 + nz,
                                      input_dtype=hf.HF_U16, z=0.3, max_batch=nwin, fftshift=shift,
                                      moment_mask=mask, form=form))
    got = p.run(ring, T * nwin, 0, nwin).cpu().numpy()
    cfg = O.PathConfig(H, W, T, T, z0, z0 + nz, z=0.3, fftshift=bool(shift))
    for w in range(nwin):
        exp = O.reconstruct_window(x[w * T:(w + 1) * T].astype(np.float64), cfg)
        for i, m in enumerate([m for m in range(3) if mask >> m & 1]):
            assert O.rel_l2(got[w, i], exp[m]) < (1e-3 if form else 1e-4), (w, m)


@pytest.mark.parametrize("H", [64, 128, 256, 512, 768, 1024])
@pytest.mark.parametrize("B", [1, 2, 17])
@pytest.mark.parametrize("mag,skip", [(True, True), (False, True), (False, False)])
def test_fresnel_column_strips(cuda, H, B, mag, skip):
    """Groups of planes in the column strips: one, full groups, a remainder; strided outputs; zeros and
    magnitudes whose squares leave float32's range."""
    import torch
    import holoflow_b200 as hf
    from holoflow_b200 import pipeline as pl
    W = 64
    rng = np.random.default_rng(H + B)
    x = _complex(rng, (B, H, W))
    exp = O.fresnel(x, LAM, DX, DX, 0.2, output_magnitude=mag, skip_phase_shift=skip)
    plan = pl.FresnelPlan(B, H, W, hf.HF_CF32, LAM, DX, 0.2, output_magnitude=mag, skip_phase_shift=skip)
    dev = torch.from_numpy(x).to(cuda)
    tol = 2e-6 * math.log2(H * W)  # the bound of the other Fresnel tests
    assert O.rel_l2(plan(dev).cpu().numpy(), exp) < tol
    out = torch.empty((H, W, B), dtype=torch.float32 if mag else torch.complex64, device=cuda).permute(2, 0, 1)
    assert O.rel_l2(plan(dev, out).cpu().numpy(), exp) < tol
    if mag:
        for scale in (1e-24, 1e30):
            assert O.rel_l2(plan(dev * scale).cpu().numpy().astype(np.float64) / scale, exp) < tol
        assert float(plan(dev * 0.0).abs().max()) == 0.0
