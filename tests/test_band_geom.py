"""Tile geometry of the FP32 band DFT (csrc/host/band_geom.hh) on the host, and on the device for the long
windows and wide bands that leave room for one or two small tiles only."""
import ctypes as C
import pathlib
import subprocess

import numpy as np
import pytest

CSRC = pathlib.Path(__file__).resolve().parents[1] / "holoflow_b200" / "csrc"
SRC = """
#include "host/band_geom.hh"
extern "C" void geom(int T, int nz, int num, int den, long long *o) {
  const hf::BandGeom g = hf::band_geom(T, nz, num, den);
  o[0] = g.NB, o[1] = g.KG, o[2] = g.nzpad, o[3] = g.stages, o[4] = (long long)g.smem;
}
// Windows that 128-pixel tiles of all frames, W padded to 14 bins and a lens row fit into 200 KB, which
// the geometry refuses: their number.
extern "C" int refused(int num, int den, int most_t) {
  int n = 0;
  for (int T = 1; T <= most_t; ++T)
    for (int nz = 1; nz <= T; ++nz) {
      const long long old = (long long)T * (128 * num / den) + (long long)T * ((nz + 13) / 14 * 14) * 8 + 128 * 8;
      n += old <= 200 * 1024 && hf::band_geom(T, nz, num, den).smem > hf::kBandSmem;
    }
  return n;
}
"""
BYTES = {"u8": (1, 1), "mono12p": (3, 2), "u16": (2, 1), "f32": (4, 1)}


@pytest.fixture(scope="module")
def geom(tmp_path_factory):
    d = tmp_path_factory.mktemp("band_geom")
    (d / "g.cc").write_text(SRC)
    subprocess.run(["g++", "-std=c++20", "-O2", "-fPIC", "-shared", "-I", str(CSRC), str(d / "g.cc"), "-o",
                    str(d / "g.so")], check=True)
    return C.CDLL(str(d / "g.so"))


@pytest.mark.parametrize("fmt", list(BYTES))
def test_no_tiled_window_is_refused(geom, fmt):
    assert geom.refused(*BYTES[fmt], 1600) == 0


@pytest.mark.parametrize("fmt", list(BYTES))
def test_groups_cover_the_bins(geom, fmt):
    o = (C.c_longlong * 5)()
    for T in (1, 2, 7, 32, 64, 100, 128, 256, 512):
        for nz in range(1, T + 1):
            geom.geom(T, nz, *BYTES[fmt], o)
            nb, kg, pad, stages, smem = o
            assert nb % 2 == 0 and 4 <= nb <= 14 and kg in (1, 2, 4) and stages in (1, 2)
            assert pad % nb == 0 and nz <= pad < nz + nb
            assert smem >= stages * T * (512 // kg) * BYTES[fmt][0] // BYTES[fmt][1] + T * pad * 8


# one stage and two beside little room, several tiles per CTA, partial tiles
@pytest.mark.gpu
@pytest.mark.parametrize("fmt,T,P,z0,z1", [("f32", 128, 40000, 0, 65), ("f32", 256, 1026, 4, 8), ("f32", 256, 20002, 4, 32),
                                           ("f32", 128, 1000, 0, 128), ("u16", 256, 1024, 4, 32), ("u16", 128, 514, 0, 128),
                                           ("u8", 512, 1030, 4, 18), ("mono12p", 512, 2050, 4, 18), ("f32", 384, 390, 0, 5)])
def test_long_windows(cuda, rng, geom, fmt, T, P, z0, z1):
    import torch
    import holoflow_b200 as hf
    from holoflow_b200 import pipeline as pl
    from oracle import oracle as O
    dt = {"u8": hf.HF_U8, "u16": hf.HF_U16, "mono12p": hf.HF_MONO12P, "f32": hf.HF_F32}[fmt]
    x = rng.integers(0, 256 if fmt == "u8" else 4096, (2, T, P))
    host = {"u8": lambda: x.astype(np.uint8), "u16": lambda: x.astype(np.uint16).view(np.int16),
            "mono12p": lambda: O.pack12(x.astype(np.uint16).reshape(-1)), "f32": lambda: x.astype(np.float32)}[fmt]()
    o = (C.c_longlong * 5)()
    geom.geom(T, z1 - z0, *BYTES[fmt], o)
    assert o[4] <= 220 * 1024
    got = pl.temporal_dft(torch.from_numpy(host).cuda(), dt, 2, T, P, z0, z1).cpu().numpy()
    assert O.rel_l2(got, np.fft.fft(x, axis=1)[:, z0:z1]) < 1e-5
