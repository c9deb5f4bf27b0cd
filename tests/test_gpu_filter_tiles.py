"""The cutoff filter's tiles: source counts on each side of a mask word, of the 128 sources that one
tensor-core product marks and of a whole tile, with targets that see many words and targets that
see none of some; pair counts against FP64 distances, forces against the walk that lists the same
leaves but filters by FP32 distances."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("leaf", [16, 48])
@pytest.mark.parametrize("n", [2, 31, 33, 127, 129, 191, 255, 256, 257, 289, 513])
def test_tiles_count_and_sum_every_pair(gpu, n, leaf):
    from scipy.spatial import cKDTree

    from blitzar_b200._lib import Engine

    rcut = 5.0 / 64
    r = np.random.default_rng(n)
    # a blob of two cutoffs across, of close pairs and a triple (a leaf of one particle, or of
    # coincident ones, would be taken as a point mass and not as a pair)
    pos = rcut * 2.0 * r.random((max(n // 2, 1), 3)) + 0.4
    pos = pos[np.minimum(np.arange(n) // 2, len(pos) - 1)] + 1e-4 * rcut * r.standard_normal((n, 3))
    pos = pos.astype(np.float32)
    m = np.full(n, 1.0 / n, np.float32)
    acc, count = {}, {}
    for order in (1, 2):
        with Engine(n, solver=1, box_length=1.0, treepm_grid_size=64, treepm_r_split_cells=1.0,
                    treepm_r_cut_factor=5.0, treepm_gradient=2, treepm_assignment=2, treepm_window_floor=0.0,
                    treepm_node_size_factor=1e-6, multipole_order=order, octree_softening=0.1 * rcut,
                    leaf_capacity=leaf, physics_max_acceleration=1e30) as e:
            e.set_state(pos, None, m)
            acc[order] = e.accelerations().astype(np.float64)
            _, count[order], nodes = e.walk_counts()
        assert nodes == 0
    tree = cKDTree(pos.astype(np.float64), boxsize=1.0)
    # (FP32 distances: 2^-24 of the coordinates, below 0.6)
    lo, hi = (tree.count_neighbors(tree, rcut + d) for d in (-3e-7, 3e-7))
    assert lo <= count[1] <= hi
    # FP32 sums of n pairs of at most m / (eps^2) each, in two orders; the FP32 mesh force is the
    # same field summed by atomics in another order
    bound = 4.0 * 2.0 ** -24 * np.sqrt(n) * m[0] / (0.1 * rcut) ** 2 * 8
    assert np.abs(acc[1] - acc[2]).max() <= bound + 1e-6 * np.abs(acc[2]).max()
