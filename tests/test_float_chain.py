"""The serial float sums that many threads evaluate (float_chain.cuh), the device functions themselves
run on the host: the bits of the sum added term by term, no term read past the last one, and a number of
steps and passes that does not grow with the terms, whatever their size and however many of them tie."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def chain(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("chain") / "chain.so")
    subprocess.run(["g++", "-std=gnu++20", "-O1", "-ffp-contract=off", "-shared", "-fPIC", "-o", so,
                    os.path.join(HERE, "float_chain_host.cpp")], check=True)
    L = C.CDLL(so)
    for f in (L.serial_weighted, L.serial_square, L.warp_weighted, L.block_square):
        f.restype = C.c_float
    return L


def _terms(kind, n, rng):
    d = rng.normal(0, 1, n)
    if kind == "nan":
        d[:] = np.nan
    elif kind == "nan-last":
        d[-1] = np.nan
    elif kind == "inf":
        d[n // 2] = np.inf
    elif kind == "ties":  # odd squares, which tie from a sum of 2^24 on
        d = rng.integers(0, 2, n) * 2 + 1.0
        d[:17] = 1001
    elif kind == "zeros":
        d[:] = 0
    elif kind != "plain":
        d *= float(kind)
    return d.astype(np.float32)


KINDS = ["plain", "ties", "zeros", "nan", "nan-last", "inf", "1e-21", "1e-24", "1e-30", "1e18", "1e22"]


def _same(a, b):
    return np.float32(a).tobytes() == np.float32(b).tobytes() or (np.isnan(a) and np.isnan(b))


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n", [1, 2, 11, 12, 13, 127, 128, 129, 700])
def test_warp(chain, kind, n):
    rng = np.random.default_rng(n)
    d, cnt = _terms(kind, n, rng), rng.integers(1, 4, n).astype(np.int32)
    last, steps = C.c_int(0), C.c_int(0)
    got = chain.warp_weighted(d.ctypes, cnt.ctypes, n, C.byref(last), C.byref(steps))
    assert last.value < n
    assert _same(got, chain.serial_weighted(d.ctypes, cnt.ctypes, n))
    # The first twelve terms, one for each binade that the rest of the sum crosses, and ties.
    assert kind == "ties" or steps.value <= 12 + 48


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n", [1, 8, 1023, 8191, 8192, 8193, 20000])
def test_block(chain, kind, n):
    d = _terms(kind, n, np.random.default_rng(n))
    barriers = C.c_int(0)
    got = chain.block_square(d.ctypes, n, C.byref(barriers))
    assert _same(got, chain.serial_square(d.ctypes, n))
    # Three barriers a pass at most: two passes a batch, and one for each binade that the sum crosses.
    assert barriers.value <= 3 * (2 * (n // 8192 + 1) + 64)
