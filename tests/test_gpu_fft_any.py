"""Any-length row and column passes (k_fft_any.cu) against the float64 oracle: edges of the radix
sets (primes with a register butterfly, larger primes through the dense stage, composite radices),
lengths around the shared-memory limit, partial row groups and strips, and every form the passes
take (real and strided input, strided output, output lens, inverse, placement in a padded plane)."""
import math

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

LAM, DX = 852e-9, 12e-6


def _tol(*sides):
    # one rounding of 2^-24 per stage level, sqrt(p) of them in a dense stage of prime p; the bound
    # of the four-step passes, 2e-6 log2(HW), covers both up to the longest length
    return 2e-6 * math.log2(math.prod(sides))


@pytest.mark.parametrize("H,W", [(2, 3), (5, 17), (19, 23), (37, 48), (90, 98), (109, 218), (480, 640), (600, 800),
                                 (601, 17), (9, 601), (387, 218), (1013, 12), (7, 2048), (2048, 5), (3, 3128),
                                 (3128, 3), (4, 3121), (2, 3200)])
@pytest.mark.parametrize("mode", ["complex", "magnitude", "phase"])
def test_fresnel_any_sides(cuda, H, W, mode):
    import torch
    import holoflow_b200 as hf
    from holoflow_b200 import pipeline as pl
    rng = np.random.default_rng(H * 10007 + W)
    B = 3
    x = (rng.standard_normal((B, H, W)) + 1j * rng.standard_normal((B, H, W))).astype(np.complex64)
    mag, skip = mode == "magnitude", mode != "phase"
    plan = pl.FresnelPlan(B, H, W, hf.HF_CF32, LAM, DX, 0.3, output_magnitude=mag, skip_phase_shift=skip)
    got = plan(torch.from_numpy(x).to(cuda)).cpu().numpy()
    exp = O.fresnel(x, LAM, DX, DX, 0.3, output_magnitude=mag, skip_phase_shift=skip)
    assert O.rel_l2(got, exp) < _tol(H, W)


def test_fresnel_any_real_strided_in_and_out(cuda):
    import torch
    import holoflow_b200 as hf
    from holoflow_b200 import pipeline as pl
    rng = np.random.default_rng(1)
    big = rng.standard_normal((2, 75, 2 * 106)).astype(np.float32)
    dev = torch.from_numpy(big).to(cuda)[:, :, ::2]
    for mag, dt in ((True, torch.float32), (False, torch.complex64)):
        plan = pl.FresnelPlan(2, 75, 106, hf.HF_F32, LAM, DX, 0.2, output_magnitude=mag)
        wide = torch.zeros((2, 75, 3 * 106), dtype=dt, device=cuda)
        plan(dev, out=wide[:, :, ::3])
        exp = O.fresnel(big[:, :, ::2], LAM, DX, DX, 0.2, output_magnitude=mag)
        w = wide.cpu().numpy()
        assert O.rel_l2(w[:, :, ::3], exp) < _tol(75, 106)
        assert not w[:, :, 1::3].any() and not w[:, :, 2::3].any()


@pytest.mark.parametrize("B,H,W,pad,real", [(2, 50, 70, None, False), (1, 33, 57, (61, 41), True),
                                            (2, 101, 37, (59, 151), False), (1, 600, 480, None, True)])
def test_angular_spectrum_any_sides(cuda, B, H, W, pad, real):
    """Forward and inverse transforms of both axes, with placement in a padded plane."""
    import torch
    import holoflow_b200 as hf
    from holoflow_b200 import pipeline as pl
    rng = np.random.default_rng(2)
    x = rng.standard_normal((B, H, W)).astype(np.float32)
    if not real:
        x = (x + 1j * rng.standard_normal((B, H, W))).astype(np.complex64)
    padding = {"width": pad[0], "height": pad[1]} if pad else None
    plan = pl.AngularSpectrumPlan(B, H, W, hf.HF_F32 if real else hf.HF_CF32, LAM, DX, 0.3, padding, None)
    got = plan(torch.from_numpy(x).to(cuda)).cpu().numpy()
    exp = O.angular_spectrum(x, LAM, DX, DX, 0.3, None, padding)
    assert O.rel_l2(got, exp) < 5e-5


def test_overflowing_squares_keep_their_magnitude(cuda):
    """|v| of values whose squares leave the float32 range, as hypot gives it."""
    import torch
    import holoflow_b200 as hf
    from holoflow_b200 import pipeline as pl
    for scale in (1e25, 1e-25):
        x = np.zeros((1, 5, 7), np.complex64)
        x[0, 2, 3] = scale
        plan = pl.FresnelPlan(1, 5, 7, hf.HF_CF32, LAM, DX, 0.3, output_magnitude=True)
        got = plan(torch.from_numpy(x).to(cuda)).cpu().numpy()
        np.testing.assert_allclose(got, np.full((1, 5, 7), scale), rtol=1e-5)


@pytest.mark.parametrize("h,w", [(2, 2), (3, 3), (16, 7), (23, 24), (34, 51), (204, 12), (255, 9), (300, 10), (607, 3),
                                 (1024, 2)])
@pytest.mark.parametrize("nz", [1, 3, 4, 5, 9])
def test_band_mean_columns(cuda, h, w, nz):
    """The sub-aperture band mean: plane groups with and without a remainder, odd and even widths (copies
    of one and two samples), strips wider than the image, columns with a dense stage."""
    import torch
    from holoflow_b200 import autofocus as af
    from oracle import shack as SH
    rng = np.random.default_rng(h + w + nz)
    x = (rng.standard_normal((nz, 2 * h, 2 * w)) + 1j * rng.standard_normal((nz, 2 * h, 2 * w))).astype(np.complex64)
    op = af.ShortTimeFresnel(x.shape, (h, w), (h, w), LAM, DX, DX, 0.25, phase_ref="global", output="mean_magnitude")
    got = op(torch.from_numpy(x).to(cuda)).cpu().numpy()
    exp = np.abs(SH.stfd(x, h, w, h, w, LAM, DX, DX, 0.25, "global", False)).mean(axis=0)
    assert O.rel_l2(got.reshape(exp.shape), exp) < 1e-5  # the bound of the other sub-aperture tests


@pytest.mark.parametrize("nz", [1, 3, 4, 9])
@pytest.mark.parametrize("prop,H,W", [("none", 7, 18), ("fresnel", 30, 50)])
def test_moments_of_a_batch(cuda, nz, prop, H, W):
    """The moment reduction of the general sizes: groups of planes and a remainder, several windows."""
    import torch
    import holoflow_b200 as hf
    from holoflow_b200 import pipeline as pl
    rng = np.random.default_rng(nz)
    T, nwin = 20, 3
    x = rng.integers(0, 4096, (T * nwin, H, W)).astype(np.uint16)
    p = pl.Pipeline(pl.PipelineConfig(height=H, width=W, frames=T, hop=T, z_begin=1, z_end=1 + nz, input_dtype=hf.HF_U16,
                                      z=0.3, max_batch=nwin,
                                      propagation=hf.HF_PROP_NONE if prop == "none" else hf.HF_PROP_FRESNEL))
    got = p.run(torch.from_numpy(x.view(np.int16)).to(cuda), T * nwin, 0, nwin).cpu().numpy()
    cfg = O.PathConfig(H, W, T, T, 1, 1 + nz, z=0.3, propagation=prop)
    for w in range(nwin):
        exp = O.reconstruct_window(x[w * T:(w + 1) * T].astype(np.float64), cfg)
        for m in range(3):
            assert O.rel_l2(got[w, m], exp[m]) < 1e-4, (w, m)
