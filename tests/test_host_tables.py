"""The library's bin tables (csrc/pp_tables.h), compiled on their own, against the
histogram's category evaluated in numpy: thresholds by bisection over all bit
patterns, the lookup over the bits of d^2, and the rule that admits the guess
from an approximate root, with the guess itself under the errors it allows."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
TOP = np.float32(np.finfo(np.float32).max).view(np.int32)

SOURCE = r"""
#include "pp_tables.h"
using namespace pp_tables;
extern "C" int pp_tables_probe(float rmin, float rincr, float rmax, int max_cells, float* T, uint16_t* lut, int cap,
                               int* n, int* shift, uint32_t* base, int* one, int* fast, double* scale) {
  Tables t;
  set_tables(t, rmin, rincr, rmax);
  const std::vector<float> th = threshold_table(t);
  std::vector<uint16_t> l;
  bool o = false;
  build_lut(th, rmax * rmax, max_cells, l, *shift, *base, &o);
  if ((int)th.size() > cap || (int)l.size() > cap) return -1;
  std::copy(th.begin(), th.end(), T);
  std::copy(l.begin(), l.end(), lut);
  *n = (int)l.size();
  *one = o;
  *fast = category_fast_ok(th, t);
  *scale = t.hscale;
  return (int)th.size();
}
"""


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    d = tmp_path_factory.mktemp("tables")
    src, lib = d / "probe.cpp", d / "probe.so"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-fPIC", "-shared", "-Wall", "-Werror",
                    "-I", os.path.join(ROOT, "paraprobe_gb300", "csrc"), str(src), "-o", str(lib)], check=True)
    f = C.CDLL(str(lib)).pp_tables_probe
    f.argtypes = [C.c_float] * 3 + [C.c_int] + [C.c_void_p] * 2 + [C.c_int] + [C.c_void_p] * 6

    def tables(rmin, rincr, rmax, max_cells=4096):
        cap = 1 << 16
        T, lut = np.zeros(cap, dtype=np.float32), np.zeros(cap, dtype=np.uint16)
        n, shift, one, fast = (C.c_int() for _ in range(4))
        base, scale = C.c_uint32(), C.c_double()
        H = f(rmin, rincr, rmax, max_cells, T.ctypes.data, lut.ctypes.data, cap, C.byref(n), C.byref(shift),
              C.byref(base), C.byref(one), C.byref(fast), C.byref(scale))
        assert H > 0
        return dict(T=T[:H], lut=lut[: n.value], shift=shift.value, base=base.value, one=bool(one.value),
                    fast=bool(fast.value), scale=scale.value, nbins=H - 2)

    return tables


def category(d2, nbins, rmin, rmax):
    """histogram::add: 0 below rmin, 1 + bin, nbins + 1 past the last bin and above rmax."""
    x = np.sqrt(np.asarray(d2, dtype=np.float32)).astype(np.float64)
    lo, hi = float(np.float32(rmin)), float(np.float32(rmax))
    scale = 1.0 / (hi - lo) * nbins if nbins else 0.0
    b = np.floor(((x - lo) * scale).astype(np.float32)).astype(np.float64)
    return np.where(x < lo, 0, np.where((x <= hi) & (b < nbins), 1 + b, nbins + 1)).astype(np.int64)


def thresholds(nbins, rmin, rmax):
    """The smallest d^2 of each category, by bisection over every finite bit pattern."""
    k = np.arange(1, nbins + 2)
    lo, hi = np.zeros(k.size, dtype=np.int64), np.full(k.size, int(TOP), dtype=np.int64)
    while np.any(lo < hi):
        mid = (lo + hi) // 2
        with np.errstate(over="ignore", invalid="ignore"):
            up = category(mid.astype(np.int32).view(np.float32), nbins, rmin, rmax) >= k
        lo, hi = np.where(up | (lo >= hi), lo, mid + 1), np.where(up & (lo < hi), mid, hi)
    return lo.astype(np.int32).view(np.float32)


SETTINGS = [(0.0, 0.01, 2.0), (0.0, 0.005, 2.0), (0.0, 0.01, 2.5), (0.0, 0.037, 1.569), (0.0, 0.0007, 0.7), (0.0, 0.4, 1.2),
            (0.0, 2.0, 2.0), (0.0, 3.0, 2.0), (0.0, 1.0 / 8192, 2.0), (0.0, 0.01, 60.0), (0.3, 0.1, 1.3), (0.05, 0.01, 1.5),
            (0.25, 0.001, 0.95), (1.9, 0.01, 2.0), (0.0, 1e-7, 2.0), (1e-3, 0.01, 2.0)]


@pytest.mark.parametrize("rmin,rincr,rmax", SETTINGS)
def test_thresholds(probe, rmin, rincr, rmax):
    t = probe(rmin, rincr, rmax)
    assert np.array_equal(t["T"][1:], thresholds(t["nbins"], rmin, rmax))


def test_thresholds_of_random_settings(probe):
    rng = np.random.default_rng(4)
    for _ in range(150):
        rmax = float(np.float32(10 ** rng.uniform(-1, 2)))
        rmin = float(np.float32(0.0 if rng.random() < 0.5 else rmax * rng.uniform(0, 0.99)))
        rincr = float(np.float32((rmax - rmin) / 10 ** rng.uniform(-0.2, 3)))
        t = probe(rmin, rincr, rmax)
        assert np.array_equal(t["T"][1:], thresholds(t["nbins"], rmin, rmax)), (rmin, rincr, rmax)


@pytest.mark.parametrize("rmin,rincr,rmax", SETTINGS)
@pytest.mark.parametrize("cells", [4096, 512, 16])
def test_lookup(probe, rmin, rincr, rmax, cells):
    """The cell's category, then up through the thresholds: one step where the
    table says that is enough."""
    t = probe(rmin, rincr, rmax, cells)
    T, H = np.append(t["T"], np.float32(np.inf)), t["nbins"] + 2
    r2 = np.float32(np.float32(rmax) * np.float32(rmax))
    rng = np.random.default_rng(5)
    bits = t["T"][1:].view(np.int32).astype(np.int64)
    near = np.clip(bits[:, None] + np.arange(-3, 4), 0, int(r2.view(np.int32))).ravel()
    d2 = np.concatenate([near.astype(np.int32).view(np.float32), (r2 * rng.random(20000)).astype(np.float32),
                         np.array([0, 1e-38, r2], dtype=np.float32)])
    assert t["lut"].size <= cells
    cell = np.clip((d2.view(np.uint32) >> t["shift"]).astype(np.int64) - t["base"], 0, t["lut"].size - 1)
    g = t["lut"][cell].astype(np.int64)
    steps = 0
    while np.any(up := (g + 1 < H) & (T[np.minimum(g + 1, H)] <= d2)):
        g += up
        steps += 1
    assert np.array_equal(g, category(d2, t["nbins"], rmin, rmax))
    if t["one"]:
        assert steps <= 1


def test_guess_is_admitted_where_it_holds(probe):
    """Bins from 0 are admitted, bins from elsewhere never; where they are, the
    guess floor(root * scale + 1/2) or the next is the category and the
    threshold decides, with the root off by 2^-23 and the product by 1/8."""
    for rmin, rincr, rmax in SETTINGS:
        t = probe(rmin, rincr, rmax)
        assert t["fast"] == (rmin == 0.0), (rmin, rincr, rmax)
        if not t["fast"]:
            continue
        T, scale = np.append(t["T"], np.float32(np.inf)), float(np.float32(t["scale"]))
        top = np.float32(np.float32(rmax) * np.float32(rmax))
        rng = np.random.default_rng(t["nbins"])
        bits = t["T"][1:].view(np.int32).astype(np.int64)
        near = np.clip(bits[:, None] + np.arange(-4, 5), 0, int(top.view(np.int32))).ravel()
        d2 = np.concatenate([near.astype(np.int32).view(np.float32), (top * rng.random(50000)).astype(np.float32)])
        want, root = category(d2, t["nbins"], rmin, rmax), np.sqrt(d2.astype(np.float64))
        for rel in (-2.0 ** -23, 0.0, 2.0 ** -23):
            for off in (-0.125, 0.0, 0.125):
                g = np.clip(np.floor(root * (1 + rel) * scale + 0.5 + off), 0, t["nbins"] + 1).astype(np.int64)
                assert np.array_equal(g + (T[g + 1] <= d2), want), (rmin, rincr, rmax)
