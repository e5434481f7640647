"""The plain FP64 path without digit words (IPT_GB300_WORDS_MAX_MB=0; very
large matrices, or no memory for them): the product extracts the digits from H
itself and has to give the bits it gives with words, at the edges of its
tiles, on rows that are not finite or far below the fast split's range, and in
FP64 block and ACX solves."""
import numpy as np
import pytest

from block_ipt_gb300 import workloads
from tests.test_gpu_fp64_fma import acx, plain
from tests.test_gpu_plain_range import SPLIT

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1), (31, 5), (33, 16), (127, 17), (128, 32), (129, 33), (257, 1), (511, 65),
          (1025, 31)]


def both(monkeypatch, call):
    words = call()
    monkeypatch.setenv("IPT_GB300_WORDS_MAX_MB", "0")
    rows = call()
    monkeypatch.delenv("IPT_GB300_WORDS_MAX_MB")
    return words, rows


def same(a, b):
    return (a.view(np.int64) == b.view(np.int64)).all()


@pytest.mark.parametrize("n,k", SHAPES)
def test_same_bits_without_words(cuda, monkeypatch, n, k):
    H = SPLIT["decay64"](n)
    a, b = both(monkeypatch, lambda: plain(cuda, H, k, 4))
    assert np.isfinite(a).all() and same(a, b)


@pytest.mark.parametrize("family", ["up", "blocks"])
def test_blocks_of_different_size(cuda, monkeypatch, family):
    H = SPLIT[family](700)
    a, b = both(monkeypatch, lambda: plain(cuda, H, 20, 3))
    assert np.isfinite(a).all() and same(a, b)


def test_rows_not_finite_and_subnormal(cuda, monkeypatch):
    rng = np.random.default_rng(5)
    n, k = 300, 18
    H = rng.standard_normal((n, n)) * 0.01
    H[40:80] *= 2.0 ** -1000
    H[np.arange(n), np.arange(n)] = np.arange(n)
    a, b = both(monkeypatch, lambda: plain(cuda, H, k, 3))
    assert np.isfinite(a).all() and same(a, b)
    H[150, 3] = np.inf
    a, b = both(monkeypatch, lambda: plain(cuda, H, k, 2))
    nan = np.isnan(a)
    assert nan.any() and (nan == np.isnan(b)).all() and (a[~nan] == b[~nan]).all()


def test_acx(cuda, monkeypatch):
    H, _ = workloads.dense_config0(777, seed=2)
    a, b = both(monkeypatch, lambda: acx(cuda, H, 12))
    assert np.isfinite(a).all() and same(a, b)
