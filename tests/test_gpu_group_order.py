"""The walk's order over its groups: group counts on each side of the sizes at which the groups are
taken by falling size (more groups than warps of a full device, and at most 32768), with equal and
with mixed group sizes; every target is written once, also by a repeated call."""
import numpy as np
import pytest

from conftest import plummer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,gsize", [(2368, 1), (2369, 1), (9000, 3), (32768, 1), (32769, 1), (60000, 9)])
def test_group_order_matches_oracle(gpu, oracle, n, gsize):
    from blitzar_b200._lib import Engine

    pos = plummer(n, seed=7 + n)
    m = (np.random.default_rng(n).random(n) + 0.5).astype(np.float32) / n
    p64 = pos.astype(np.float64)
    lo = p64.min(0)
    keys = oracle.morton63(p64, lo, float((p64.max(0) - lo).max()))
    perm = oracle.stable_sort(keys)
    sp4 = oracle.pos4(pos[perm], m[perm])
    tree = oracle.build_tree(keys[perm], sp4, leaf_cap=16)
    w = oracle.walk(sp4, tree, theta=0.9, eps=0.01, quadrupole=True, want_pot=True, gmax=gsize)
    with Engine(n, octree_theta=0.9, octree_softening=0.01, multipole_order=2, walk_group_size=gsize,
                physics_max_acceleration=1e30) as e:
        e.set_state(pos, None, m)
        acc = e.accelerations()
        npp, npn = e.interaction_counts()
        acc_p, pot = e.accelerations(want_pot=True)
        again, pot2 = e.accelerations(want_pot=True)
    assert npp == int((w["n_pp"] * w["group_sizes"]).sum())
    assert npn == int((w["n_pn"] * w["group_sizes"]).sum())
    # FP32 sums of at most n terms: the walk's parity bound, 1e-5 of the net force
    scale = np.linalg.norm(w["acc"], axis=1)
    for a in (acc, acc_p):
        assert (np.linalg.norm(a[perm].astype(np.float64) - w["acc"], axis=1) / scale).max() < 1e-5
    assert np.abs(pot[perm] - w["pot"]).max() <= 1e-5 * np.abs(w["pot"]).max()
    assert np.array_equal(acc_p, again) and np.array_equal(pot, pot2)
