"""The all-levels-at-once topology and the small sort by counting at the sizes where they can go wrong:
around block and run sizes, leaf capacities from one particle to more than the system holds,
duplicates down to the depth limit, and a node count past the array's capacity."""
import numpy as np
import pytest

from conftest import plummer

pytestmark = pytest.mark.gpu


def _tree(n, pos, m, **kw):
    from blitzar_b200._lib import Engine

    with Engine(n, physics_max_acceleration=1e30, **kw) as e:
        e.set_state(pos, None, m)
        keys, perm = e.morton_keys()
        return e.tree(), keys, perm


@pytest.mark.parametrize("n", [1, 2, 31, 511, 512, 513, 1024, 1025, 4096, 4097, 8192, 8193, 20_001])
@pytest.mark.parametrize("leaf", [1, 5, 16, 300, 100_000])
def test_topology_and_order_match_oracle(gpu, oracle, n, leaf):
    rng = np.random.default_rng(n + leaf)
    pos = plummer(n, seed=n)
    pos[rng.random(n) < 0.1] = pos[0]  # identical keys (at most 10 %): ties and the depth limit
    m = (rng.random(n) + 0.5).astype(np.float32) / n
    p64 = pos.astype(np.float64)
    lo = p64.min(0)
    keys = oracle.morton63(p64, lo, float((p64.max(0) - lo).max()) or 1.0)
    perm = oracle.stable_sort(keys)
    o = oracle.build_tree(keys[perm], oracle.pos4(pos[perm], m[perm]), leaf_cap=leaf)
    t, k, p = _tree(n, pos, m, leaf_capacity=leaf)
    assert np.array_equal(k, keys[perm]) and np.array_equal(p, perm)
    assert t["nodes"] == o["nodes"]
    for name in ("start", "count", "child", "nchild", "mono", "bmin", "bmax", "quad"):
        assert np.array_equal(t[name], o[name]), name


@pytest.mark.parametrize("n", [600_001, (1 << 20) - 1, (1 << 20) + 1, (1 << 23) - 1, (1 << 23) + 4097])
def test_topology_of_large_systems(gpu, oracle, n):
    """2, 4 and 16 particles a thread, and scans of more than 1024 block counts."""
    pos = plummer(n, seed=n)
    pos[:: n // 40] = pos[0]
    m = np.full(n, 1.0 / n, np.float32)
    p64 = pos.astype(np.float64)
    lo = p64.min(0)
    keys = oracle.morton63(p64, lo, float((p64.max(0) - lo).max()))
    perm = oracle.stable_sort(keys)
    o = oracle.build_tree(keys[perm], oracle.pos4(pos[perm], m[perm]), leaf_cap=16)
    t, k, p = _tree(n, pos, m, leaf_capacity=16)
    assert np.array_equal(k, keys[perm]) and np.array_equal(p, perm)
    assert t["nodes"] == o["nodes"]
    for name in ("start", "count", "child", "nchild", "mono", "bmin", "bmax", "quad"):
        assert np.array_equal(t[name], o[name]), name


def test_node_capacity_overflow_is_reported(gpu):
    """Close pairs far apart need a chain of single-child nodes each: more nodes than the arrays
    hold.  The build stops at the last level that fits and reports the limit."""
    from blitzar_b200._lib import BZ_DEVICE_LIMIT, BzError, Engine

    n = 20_000
    rng = np.random.default_rng(3)
    base = rng.random((n // 2, 3))
    pos = np.concatenate([base, base + 1e-6])
    with Engine(n, leaf_capacity=1, octree_theta=1.0, physics_max_acceleration=1e30) as e:
        e.set_state(pos, None, np.full(n, 1.0 / n, np.float32), f64=True)
        with pytest.raises(BzError) as err:
            e.accelerations()
        assert err.value.status == BZ_DEVICE_LIMIT
        e.set_state(plummer(n, seed=4), None, np.full(n, 1.0 / n, np.float32))
        assert np.isfinite(e.accelerations()).all()  # the handle goes on
