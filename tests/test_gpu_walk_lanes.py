"""The walk's sharing of a group's targets over the 32 lanes: group sizes on each side of every
slot count (1, 2 and 4 slots, odd and even rows), list lengths from one entry to many flushes, the
packed and the guarded pair laws, forces and potentials against the oracle's FP64 walk."""
import numpy as np
import pytest

from conftest import plummer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 33, 700, 9001])
@pytest.mark.parametrize("gsize", [1, 2, 3, 4, 5, 8, 9, 31, 32])
def test_lane_shares_match_oracle(gpu, oracle, n, gsize):
    from blitzar_b200._lib import Engine

    pos = plummer(n, seed=100 + n)
    m = (np.random.default_rng(n).random(n) + 0.5).astype(np.float32) / n
    p64 = pos.astype(np.float64)
    lo = p64.min(0)
    keys = oracle.morton63(p64, lo, float((p64.max(0) - lo).max()) or 1.0)
    perm = oracle.stable_sort(keys)
    sp4 = oracle.pos4(pos[perm], m[perm])
    tree = oracle.build_tree(keys[perm], sp4, leaf_cap=16)
    # eps below the minimum distance 1e-6 takes the guarded pair law, above it the packed one
    for eps in (0.01, 1e-8):
        for order in (2, 1):
            w = oracle.walk(sp4, tree, theta=0.5, eps=eps, quadrupole=order == 2, want_pot=True, gmax=gsize)
            with Engine(n, octree_theta=0.5, octree_softening=eps, multipole_order=order, walk_group_size=gsize,
                        physics_max_acceleration=1e30) as e:
                e.set_state(pos, None, m)
                acc = e.accelerations()[perm].astype(np.float64)
                npp, npn = e.interaction_counts()
                acc_p, pot = e.accelerations(want_pot=True)
            assert npp == int((w["n_pp"] * w["group_sizes"]).sum())
            assert npn == int((w["n_pn"] * w["group_sizes"]).sum())
            # FP32 sums of at most n terms: the walk's parity bound, 1e-5 of the net force
            scale = np.maximum(np.linalg.norm(w["acc"], axis=1), 1e-30)
            for a in (acc, acc_p[perm].astype(np.float64)):
                assert (np.linalg.norm(a - w["acc"], axis=1) / scale).max() < 1e-5
            assert np.abs(pot[perm] - w["pot"]).max() <= 1e-5 * np.abs(w["pot"]).max() + 1e-30
