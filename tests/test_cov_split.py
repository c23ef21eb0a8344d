"""CTA split and workspace of the Gram matrices (csrc/host/cov_split.hh) on the host: a plan makes its
workspace once, for max_batch windows, and every call of fewer windows has to fit in it."""
import ctypes as C
import pathlib
import subprocess

import pytest

CSRC = pathlib.Path(__file__).resolve().parents[1] / "holoflow_b200" / "csrc"
SRC = """
#include "host/cov_split.hh"
extern "C" long long split(int sms, long long nt, int n) { return hf::cov_split(sms, nt, n); }
extern "C" long long most(int sms, long long nt, int n) { return hf::cov_split_most(sms, nt, n); }
// The first call of 1 .. most_windows windows that does not fit a plan of some max_batch, or 0.
extern "C" int first_overflow(int sms, long long nt, int most_windows) {
  long long need = 0;
  for (int b = 1; b <= most_windows; ++b) {
    const long long n = b * hf::cov_split(sms, nt, b);
    need = n > need ? n : need;
    if (need > hf::cov_split_most(sms, nt, b))
      return b;
  }
  return 0;
}
"""


@pytest.fixture(scope="module")
def split(tmp_path_factory):
    d = tmp_path_factory.mktemp("cov_split")
    (d / "s.cc").write_text(SRC)
    subprocess.run(["g++", "-std=c++20", "-O2", "-fPIC", "-shared", "-I", str(CSRC), str(d / "s.cc"), "-o",
                    str(d / "s.so")], check=True)
    lib = C.CDLL(str(d / "s.so"))
    for f in (lib.split, lib.most):
        f.restype, f.argtypes = C.c_longlong, [C.c_int, C.c_longlong, C.c_int]
    lib.first_overflow.argtypes = [C.c_int, C.c_longlong, C.c_int]
    return lib


@pytest.mark.parametrize("tiles", [1, 2, 9, 16, 64, 100, 400, 8192])
@pytest.mark.parametrize("sms", [1, 132, 148])
def test_every_smaller_call_fits_the_workspace(split, sms, tiles):
    assert split.first_overflow(sms, tiles, 4096) == 0


def test_split_covers_at_most_the_tiles(split):
    for n in (1, 2, 7, 36, 37, 148, 296, 297, 5000):
        for nt in (1, 3, 64, 10000):
            assert 1 <= split.split(148, nt, n) <= nt


def test_per_window_workspace_times_the_batch(split):
    """hf_covariance: one window's workspace per batch item holds the whole batch."""
    for nt in (1, 5, 64, 400):
        for n in (1, 2, 7, 36, 147, 148, 1000):
            assert n * split.split(148, nt, n) <= n * split.most(148, nt, 1)


@pytest.mark.gpu
@pytest.mark.parametrize("side,T,max_batch,nwin", [(64, 50, 37, 36), (160, 32, 148, 147), (64, 32, 33, 32)])
def test_fewer_windows_than_max_batch(cuda, rng, side, T, max_batch, nwin):
    import numpy as np
    import torch
    import holoflow_b200 as hf
    from holoflow_b200 import pipeline as pl
    n = T + nwin - 1
    x = rng.integers(0, 4096, (n, side * side)).astype(np.uint16)
    cfg = pl.PipelineConfig(side, side, T, 1, 1, 3, input_dtype=hf.HF_U16, clutter_rank=2, max_batch=max_batch)
    p = pl.Pipeline(cfg)
    p.run(torch.from_numpy(x.view(np.int16)).cuda(), n, 0, nwin)
    for w in (0, nwin // 2, nwin - 1):
        gram, _ = p.inspect(w)
        X = x[w:w + T].astype(np.float64)
        G = X @ X.T
        assert np.abs(gram.cpu().numpy() - G).max() / G.max() < 2e-7
