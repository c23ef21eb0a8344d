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


@pytest.mark.parametrize("W", [256, 257 * 2])  # 512 tiles in one CTA; a few more: two CTAs per window
def test_integer_gram_accumulator_range(cuda, W):
    """As many windows as the GPU has SMs and full-scale samples: the largest sums a CTA accumulates."""
    import torch
    import holoflow_b200 as hf
    from holoflow_b200 import pipeline as pl
    T, hop, H = 128, 8, 256 if W == 256 else 128
    nwin = torch.cuda.get_device_properties(0).multi_processor_count
    n, P = T + hop * (nwin - 1), H * W
    ring = torch.full((n * P * 3 // 2,), 255, dtype=torch.uint8, device=cuda)
    ring[7 * P * 3 // 2:8 * P * 3 // 2] = 0  # frame 7 of the first window
    p = pl.Pipeline(pl.PipelineConfig(height=H, width=W, frames=T, hop=hop, z_begin=1, z_end=2, input_dtype=hf.HF_MONO12P,
                                      propagation=hf.HF_PROP_NONE, clutter_rank=1, max_batch=nwin, form=1))
    p.run(ring, n, 0, nwin)
    for w in (0, 1, nwin - 1):
        gram, _ = p.inspect(w)
        exp = np.full((T, T), float(P * 4095 * 4095))
        if w == 0:
            exp[7, :] = exp[:, 7] = 0.0
        assert np.array_equal(gram.cpu().numpy(), exp), w


def _check_pairs(a, ev, V, r):
    n = a.shape[0]
    scale = np.abs(a).max()
    w = np.linalg.eigvalsh(a / scale)[n - r:]
    assert np.abs(ev / scale - w).max() < 1e-12 * n  # eigenvalues to the rounding of ||A||
    assert np.abs(V.T @ V - np.eye(r)).max() < 1e-12
    assert np.abs((a / scale) @ V - V * (ev / scale)).max() < 1e-12 * n


@pytest.mark.parametrize("n", [1, 2, 3, 4, 20, 21, 33, 64, 65, 128])
@pytest.mark.parametrize("kind", ["gram", "tiny", "huge", "rank1", "diagonal", "blocks", "zero"])
def test_eigensolver_limits(cuda, n, kind):
    """Entries near both ends of the exponent range, decoupled and degenerate spectra."""
    import torch
    from holoflow_b200 import pipeline as pl
    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, 3 * n)) + 10.0
    a = x @ x.T
    if kind == "tiny":
        a = a * 1e-280
    elif kind == "huge":
        a = a * 1e280
    elif kind == "rank1":
        a = np.outer(x[:, 0], x[:, 0])
    elif kind == "diagonal":
        a = np.diag(np.repeat(np.arange(1.0, n + 1), 2)[:n])
    elif kind == "blocks":
        a[: n // 2, n // 2:] = 0.0
        a[n // 2:, : n // 2] = 0.0
    elif kind == "zero":
        a = np.zeros((n, n))
    r = min(n, 4)
    ev, V, info = pl.eigh_top(torch.from_numpy(np.stack([a, a])).to(cuda), r)
    assert info.cpu().tolist() == [0, 0]
    ev, V = ev.cpu().numpy(), V.cpu().numpy()
    assert np.array_equal(ev[0], ev[1]) and np.array_equal(V[0], V[1])
    if kind == "zero":
        assert np.abs(ev).max() < 1e-300 + 1e-15
        assert np.abs(V[0].T @ V[0] - np.eye(r)).max() < 1e-12
    else:
        _check_pairs(a, ev[0], V[0], r)


@pytest.mark.parametrize("T,rank,z0,z1", [(7, 0, 0, 7), (64, 4, 4, 32), (128, 1, 0, 64), (128, 60, 3, 67),
                                          (128, 100, 0, 128), (33, 5, 1, 2)])
def test_band_matrix_staged_and_direct(cuda, T, rank, z0, z1):
    import torch
    import holoflow_b200 as hf
    from holoflow_b200 import pipeline as pl
    rng = np.random.default_rng(T)
    V = np.stack([np.linalg.qr(rng.standard_normal((T, T)))[0] for _ in range(2)])
    dev = torch.from_numpy(V).to(cuda)
    w = torch.empty((2, T, z1 - z0), dtype=torch.complex64, device=cuda)
    hf.check(hf.lib().hf_band_matrix(pl._ptr(dev), 2, T, rank, z0, z1, pl._ptr(w), pl._stream()))
    for b in range(2):
        exp = O.band_matrix(T, z0, z1, V[b][:, T - rank:])
        assert np.abs(w[b].cpu().numpy() - exp).max() < 2.0 ** -22 * np.abs(exp).max() + 1e-14


@pytest.mark.parametrize("fmt", ["u8", "u16", "f32", "mono12p"])
@pytest.mark.parametrize("T,P", [(1, 64), (7, 30), (8, 257), (16, 4098), (33, 1000), (50, 2050), (64, 4096), (100, 514),
                                 (128, 3002), (130, 66)])
def test_fp32_gram_any_length_and_alignment(cuda, fmt, T, P):
    """Block edges, ragged tiles, rows of any alignment; with and without a workspace."""
    import torch
    import holoflow_b200 as hf
    from holoflow_b200 import pipeline as pl
    if fmt == "mono12p" and P % 2:
        pytest.skip("packed frames have an even pixel count")
    rng = np.random.default_rng(T * P)
    top = {"u8": 256, "u16": 65536, "f32": 4096, "mono12p": 4096}[fmt]
    x = rng.integers(0, top, (2, T, P))
    if fmt == "mono12p":
        raw, dt = O.pack12(x.astype(np.uint16).reshape(-1)), hf.HF_MONO12P
    else:
        raw, dt = {"u8": (x.astype(np.uint8).reshape(-1), hf.HF_U8),
                   "u16": (x.astype(np.uint16).reshape(-1).view(np.uint8), hf.HF_U16),
                   "f32": (x.astype(np.float32).reshape(-1).view(np.uint8), hf.HF_F32)}[fmt]
    for off in (0, 4):
        buf = torch.zeros(raw.size + off, dtype=torch.uint8, device=cuda)
        buf[off:] = torch.from_numpy(raw.copy()).to(cuda)
        dev = buf[off:]
        got = [pl.covariance(dev, dt, 2, T, P).cpu().numpy()]
        noalloc = torch.empty((2, T, T), dtype=torch.float64, device=cuda)
        got.append(pl.covariance_noalloc(dev, dt, 2, T, P, noalloc).cpu().numpy())
        for g in got:
            for b in range(2):
                X = x[b].astype(np.float64)
                exp = X @ X.T
                assert np.abs(g[b] - exp).max() / np.abs(exp).max() < 2e-7
                assert np.array_equal(g[b], g[b].T)
