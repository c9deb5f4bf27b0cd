"""The learned correction's dense pair tiles, target by target: (accelerations with the correction) minus
(without) against a host sum over the FP64 neighbour pairs of the oracle's network.  Clusters of 1 to 64
particles (a target's pairs include itself) make runs that begin and end anywhere in a warp and in a
128-row tile and last batches that are not full; one system is large enough for batches of 64 targets."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _params(seed, flat):
    """flat: rows of almost the same output (b3 of order 1, a weak network), so that a row too many or
    too few, or the mass of a wrong source, stands out of the BF16 rounding."""
    rng = np.random.default_rng(seed)
    p = np.zeros(1667, np.float32)
    p[0:512] = rng.uniform(-0.5, 0.5, 512)
    p[512:1536] = rng.uniform(-0.3, 0.3, 1024)
    p[1536:1568] = rng.uniform(-0.1, 0.1, 32)
    p[1568:1664] = rng.uniform(-0.4, 0.4, 96) * (0.02 if flat else 1.0)
    p[1664:1667] = (1.0, -1.5, 0.75) if flat else rng.uniform(-0.1, 0.1, 3)
    return p


def _clusters(sizes, cells, spread, seed):
    """Clusters around the centres of the first octree cells of a level (cells a side), each inside its
    cell, so that a leaf is a whole cluster; particles in random caller order."""
    rng = np.random.default_rng(seed)
    at = rng.permutation(cells ** 3)[: len(sizes)]
    centre = (np.stack(np.unravel_index(at, (cells,) * 3), -1) + 0.5) / cells
    pos = np.repeat(centre, sizes, 0) + spread * rng.uniform(-1, 1, (int(np.sum(sizes)), 3))
    return pos[rng.permutation(len(pos))].astype(np.float32)


def _rows(params, pos, mass, targets, mesh, radius):
    """Correction of each target, the sum of its rows' magnitudes and its number of rows; None for one
    with a pair within 1e-5 of the radius."""
    from scipy.spatial import cKDTree

    from oracle import oracle

    p = pos.astype(np.float64)
    tree = cKDTree(p, boxsize=1.0)
    near = tree.query_ball_point(p[targets], radius * (1 + 1e-5) / mesh)
    inner = tree.query_ball_point(p[targets], radius * (1 - 1e-5) / mesh, return_length=True)
    tgt, src = np.repeat(targets, [len(s) for s in near]), np.concatenate([np.asarray(s, int) for s in near])
    d = p[tgt] - p[src]
    d -= np.rint(d)
    x = np.concatenate([d * mesh, p[src] * mesh % 1.0], 1).astype(np.float32)
    out = oracle.mlp_forward(params, x, 0.5).astype(np.float64) * (mass[src].astype(np.float64) * mesh ** 2)[:, None]
    for k, t in enumerate(targets):
        own = out[tgt == t] if len(targets) < 2000 else None
        if own is None:
            raise AssertionError("too many targets for this search")
        yield t, None if len(own) != inner[k] else (-own.sum(0), np.linalg.norm(own, axis=1).sum(), len(own))


def _difference(pos, mass, params, mesh, **kw):
    from blitzar_b200._lib import Engine

    cfg = dict(solver=1, box_length=1.0, treepm_grid_size=mesh, treepm_r_split_cells=1.0, treepm_r_cut_factor=5.0,
               treepm_assignment=2, treepm_gradient=2, treepm_window_floor=0.0, treepm_node_size_factor=1e-6,
               octree_softening=0.5 / mesh, leaf_capacity=64, physics_max_acceleration=1e30)
    cfg.update(kw)
    with Engine(len(pos), **cfg) as e:
        e.set_state(pos, None, mass)
        plain = e.accelerations().astype(np.float64)
        e.learn_set(params, 0.5)
        e.learn_enable(True)
        return e.accelerations().astype(np.float64) - plain, np.abs(plain).max()


SIZES = ([1, 64, 63, 2, 33, 32, 31, 64, 64, 1, 1, 1, 5, 17, 60, 64, 3, 48],
         [64] * 9 + [1],
         [1] * 40,
         [1],
         [2],
         [31, 33] * 12,
         list(range(1, 61)))


@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("flat", [True, False])
@pytest.mark.parametrize("case", range(len(SIZES)))
def test_rows_of_every_target(gpu, oracle, case, flat, order):
    sizes = SIZES[case]
    mesh, radius = 32, 5.0
    pos = _clusters(sizes, 4, 0.02, 10 + case)
    n = len(pos)
    mass = ((np.random.default_rng(case).random(n) + 0.5) / n).astype(np.float32)
    params = _params(case, flat)
    diff, biggest = _difference(pos, mass, params, mesh, multipole_order=order)
    rows = dict(_rows(params, pos, mass, np.arange(n), mesh, radius))
    assert sorted(r[2] for r in rows.values()) == sorted(np.repeat(sizes, sizes))
    err = np.array([np.linalg.norm(diff[t] - r[0]) - 8 * 2.0 ** -23 * biggest for t, r in rows.items()])
    mag = np.array([r[1] for r in rows.values()])
    # BF16 activations (2^-9 each, two layers; the oracle has the same rounding points, so ties and FP32
    # sums are all that differs): 3e-2 of a single row at most, as the forward pass's test allows; of
    # nearly equal rows 1/64 = 1.6e-2 is one row, and the weak network's part of them is 0.02 of that 3e-2
    assert np.all(err < (1.5e-3 if flat else 3e-2) * mag), (err / mag).max()
    assert np.median(err / mag) < (1e-4 if flat else 2e-3)


def test_batches_of_64_targets(gpu, oracle):
    """At least 8 batches of 64 targets for each of 8 blocks an SM: 610,000 particles on 148 SMs."""
    import torch

    mesh = 128
    sizes = np.full(64 ** 3, 2)
    sizes[:86_007] = 3
    n = int(sizes.sum())
    assert n >= 8 * 64 * 8 * torch.cuda.get_device_properties(0).multi_processor_count and n % 64 != 0
    pos = _clusters(sizes, 64, 0.15 / 64, 3)
    mass = ((np.random.default_rng(4).random(n) + 0.5) / n).astype(np.float32)
    params = _params(5, True)
    # the engine's radius: 5 cells, or as many as hold 25.6 neighbours at the mean density
    radius = min(5.0, (0.4 * 64 / (4.0 / 3.0 * np.pi * n / mesh ** 3)) ** (1.0 / 3.0))
    diff, biggest = _difference(pos, mass, params, mesh, leaf_capacity=8, multipole_order=1)
    targets = np.unique(np.concatenate([[0, n - 1], np.random.default_rng(6).integers(0, n, 1500)]))
    checked = 0
    for t, r in _rows(params, pos, mass, targets, mesh, radius):
        if r is not None:
            assert r[2] <= 64
            assert np.linalg.norm(diff[t] - r[0]) < 1.5e-3 * r[1] + 8 * 2.0 ** -23 * biggest, t
            checked += 1
    assert checked > 1400
