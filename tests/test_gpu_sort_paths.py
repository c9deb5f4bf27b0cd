"""The adaptive sort on every path that a system's size and order can take, bit for bit against the
oracle's stable sort: full sorts on each side of the tile length's switch (2^19 pairs) and of the chunks'
(2^20), and re-sorts whose out-of-order pairs are just few enough to be ranked by counting (4096), one
more, as many as the fast path takes (an eighth of the pairs), and one more than that."""
import numpy as np
import pytest

from conftest import plummer
from test_gpu_keys_sort import _fast_path

pytestmark = pytest.mark.gpu

SMALL_F = 4096


def _order(oracle, pos):
    p = pos.astype(np.float64)
    lo = p.min(0)
    keys = oracle.morton63(p, lo, float((p.max(0) - lo).max()))
    return keys, oracle.stable_sort(keys)


def _out_of_order(k, window=8):
    f = np.zeros(len(k), bool)
    for w in range(1, window + 1):
        f[w:] |= k[w:] < k[:-w]
        f[:-w] |= k[:-w] > k[w:]
    return int(f.sum())


def _displaced(keys, order, count):
    """Sorted order with exactly `count` positions out of order: swapped neighbours (two each) and, for an
    odd count, one run of three rotated."""
    idx = order.copy()
    k = keys[order]
    at = np.flatnonzero((k[1:-1] < k[2:]) & (k[:-2] < k[1:-1]))  # (three different keys from here)
    at = at[(at % 3 == 0) & (at + 4 < len(k))]
    if count % 2:
        j = at[-1]
        idx[j:j + 3] = idx[j + 1], idx[j + 2], idx[j]
        at = at[:-2]
        count -= 3
    at = at[np.linspace(0, len(at) - 1, count // 2).astype(int)]
    assert len(np.unique(at)) == count // 2
    idx[at], idx[at + 1] = idx[at + 1].copy(), idx[at].copy()
    return idx


def _check(oracle, pos):
    from blitzar_b200._lib import Engine

    keys, order = _order(oracle, pos)
    n = len(pos)
    with Engine(n) as e:
        e.set_state(pos, None, np.full(n, 1.0 / n, np.float32))
        got, perm = e.morton_keys()
    assert np.array_equal(perm, order)
    assert np.array_equal(got, keys[order])


@pytest.mark.parametrize("n", [8193, (1 << 19) - 1, 1 << 19, (1 << 19) + 1, (1 << 20) - 1, (1 << 20) + 4099, 3_000_001])
def test_full_sort_at_the_size_switches(gpu, oracle, n):
    pos = plummer(n, seed=n)
    pos[::37] = pos[0]  # ties: stable order
    keys, _ = _order(oracle, pos)
    assert not _fast_path(keys)
    _check(oracle, pos)


@pytest.mark.parametrize("n", [8193, 40_001, (1 << 19) + 1, (1 << 20) - 1, (1 << 20) + 4099])
@pytest.mark.parametrize("count", [0, 2, 4095, SMALL_F, SMALL_F + 1, "cap", "cap + 1"])
def test_resort_at_the_limits(gpu, oracle, n, count):
    cap = max(n // 8, SMALL_F)
    count = {"cap": cap, "cap + 1": cap + 1}.get(count, count)
    if count > cap + 1:
        count = cap + 1
    pos = plummer(n, seed=n)
    keys, order = _order(oracle, pos)
    idx = _displaced(keys, order, count)
    assert _out_of_order(keys[idx]) == count
    assert _fast_path(keys[idx]) == (count <= cap)
    _check(oracle, pos[idx])
