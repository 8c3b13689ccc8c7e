"""Ray arithmetic of the traversal (porerad_b200/csrc/pr_math.cuh) on the host, bit for bit against the
operations it replaces: the double-double sine and cosine, the division by the vector's length, and
the quotients of the first crossings."""

from __future__ import annotations

import ctypes
import subprocess

import numpy as np
import pytest

from tests.helpers import ROOT

N = 2_000_000


@pytest.fixture(scope="module")
def ht(tmp_path_factory):
    out = tmp_path_factory.mktemp("ht") / "libht.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-march=native", "-ffp-contract=off", "-fno-fast-math", "-fPIC",
                    "-shared", str(ROOT / "tests" / "host_trace_math_harness.cpp"), "-o", str(out), "-lm"], check=True)
    lib = ctypes.CDLL(str(out))
    vp, n = ctypes.c_void_p, ctypes.c_long
    lib.ht_sincos.argtypes = [vp, n, vp, vp, vp, vp]
    lib.ht_unit.argtypes = [vp, n]
    lib.ht_div.argtypes = [vp, vp, n, vp]
    return lib


def _uniforms(rng, n):
    return rng.integers(0, 1 << 53, n).astype(np.float64) * 2.0**-53


def _azimuths(kind, rng):
    if kind == "uniform":
        u = _uniforms(rng, N)
    else:  # within 2^40 units of the table's nodes, where sine or cosine vanishes among them
        u = rng.integers(0, 129, N) / 128.0 + rng.integers(-(1 << 40), 1 << 40, N) * 2.0**-53 * 2.0**-rng.integers(0, 40, N)
        u = u[(u >= 0) & (u < 1)]
        u = np.floor(u * 2.0**53) * 2.0**-53
    return (2.0 * np.pi) * u


@pytest.mark.parametrize("kind", ["uniform", "nodes"])
def test_sincos_equals_the_series(ht, kind):
    x = _azimuths(kind, np.random.default_rng(3))
    x[:2] = 0.0, (2.0 * np.pi) * (1 - 2.0**-53)
    out = np.empty((4, x.size))
    ht.ht_sincos(x.ctypes.data, x.size, *(o.ctypes.data for o in out))
    assert np.array_equal(out[0], out[2]) and np.array_equal(out[1], out[3])


@pytest.mark.parametrize("kind", ["uniform", "grazing", "normal", "scaled"])
def test_unit_vector_equals_the_divisions(ht, kind):
    rng = np.random.default_rng(5)
    u, a = _uniforms(rng, N), (2.0 * np.pi) * _uniforms(rng, N)
    if kind == "grazing":
        u = 1.0 - u * 2.0**-40
    if kind == "normal":
        u = u * 2.0**-40
    r = np.sqrt(u)
    v = np.stack((np.sqrt(1.0 - u), r * np.cos(a), r * np.sin(a)), axis=1)
    if kind == "scaled":  # lengths up to 1000 units from one, and others
        v *= 1.0 + rng.integers(-500, 500, N)[:, None] * 2.0**-52
        v[::3] *= rng.uniform(0.5, 2.0, v[::3].shape[0])[:, None]
    length = np.sqrt((v[:, 0] * v[:, 0] + v[:, 1] * v[:, 1]) + v[:, 2] * v[:, 2])
    want = v / length[:, None]
    got = np.ascontiguousarray(v)
    ht.ht_unit(got.ctypes.data, N)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("kind", ["uniform", "small divisors", "near one"])
def test_quotients_equal_the_division(ht, kind):
    rng = np.random.default_rng(7)
    b = _uniforms(rng, N) + 2.0**-53
    a = np.maximum(_uniforms(rng, N), 1.0e-12)
    if kind == "small divisors":
        b *= 2.0 ** -rng.integers(0, 60, N)
    if kind == "near one":
        b = 1.0 - rng.integers(0, 4096, N) * 2.0**-53
        a = 1.0 - rng.integers(0, 4096, N) * 2.0**-53
    a[:3] = 0.0, 1.0, 1.0e-12
    q = np.empty(N)
    ht.ht_div(a.ctypes.data, b.ctypes.data, N, q.ctypes.data)
    assert np.array_equal(q, a / b)
