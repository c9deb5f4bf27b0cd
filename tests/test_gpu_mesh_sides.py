"""The periodic mesh solve at every side the fused z transform is built for and one on each side of
them, against the same Green's function applied in FP64; and the tensor-core cutoff filter's pair
counts against the FP64 distances."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mesh", [32, 64, 128, 256, 512])
@pytest.mark.parametrize("gradient,assign", [(0, 0), (2, 2)])
def test_potential_matches_fp64_solve(gpu, mesh, gradient, assign):
    from blitzar_b200._lib import Engine

    rng = np.random.default_rng(mesh)
    n, rs = 20_000, 1.1
    with Engine(n, solver=1, box_length=1.0, treepm_grid_size=mesh, treepm_r_split_cells=rs, treepm_assignment=assign,
                treepm_gradient=gradient, treepm_window_floor=0.08) as e:
        e.set_state(rng.random((n, 3)), None, ((rng.random(n) + 0.5) / n).astype(np.float32), f64=True)
        rho = e.pm_mesh(0).reshape(mesh, mesh, mesh).astype(np.float64)
        phi = e.pm_mesh(1).reshape(mesh, mesh, mesh)
    k = 2 * np.pi * np.fft.fftfreq(mesh, 1 / mesh)
    kr = 2 * np.pi * np.fft.rfftfreq(mesh, 1 / mesh)
    k2 = k[:, None, None] ** 2 + k[None, :, None] ** 2 + kr[None, None, :] ** 2
    s, sr = np.sinc(k / (2 * np.pi * mesh)), np.sinc(kr / (2 * np.pi * mesh))
    window = (s[:, None, None] * s[None, :, None] * sr[None, None, :]) ** (2 * (assign + 2))
    k2[0, 0, 0] = 1.0
    green = 4 * np.pi * np.exp(-k2 * (rs / mesh) ** 2) / (k2 * np.maximum(window, 0.08))
    green[0, 0, 0] = 0.0
    ref = np.fft.irfftn(np.fft.rfftn(rho) * green, s=rho.shape, axes=(0, 1, 2))
    # two FP32 transforms of M^3 points: a few 2^-24 sqrt(log2 M^3) of the norm, far below 2e-6
    assert np.linalg.norm(phi - ref) < 2e-6 * np.linalg.norm(ref)


def _pairs_box(side, shift, seed):
    """Jittered lattice of close pairs: no octree leaf (at 16 a leaf) holds a single particle, which
    the walk would take as a point mass and not as a pair."""
    rng = np.random.default_rng(seed)
    g = (np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3) + 0.5) / side
    p = g + 0.2 / side * rng.standard_normal(g.shape) + shift
    pos = (np.concatenate([p, p + 1e-4 / side * rng.standard_normal(g.shape)]) % 1.0).astype(np.float32)
    pos[pos >= 1.0] = 0.0
    return pos


@pytest.mark.parametrize("rcf", [0.3, 4.5, 5.0])
@pytest.mark.parametrize("side,shift,seed", [(16, 0.0, 1), (12, 0.4999, 1), (21, 0.3, 2)])
def test_cutoff_filter_counts_every_pair(gpu, rcf, side, shift, seed):
    """Pairs through the pair law of a walk that only filters = pairs inside the cutoff, whether the
    group is far wider than the cutoff (scalar filter) or not; FP64 distances of the FP32 positions,
    pairs within 2e-6 of the cutoff (rounding of a periodic image) left open."""
    from scipy.spatial import cKDTree

    from blitzar_b200._lib import Engine

    pos = _pairs_box(side, shift, seed)
    n = len(pos)
    with Engine(n, solver=1, box_length=1.0, treepm_grid_size=64, treepm_r_split_cells=1.0, treepm_r_cut_factor=rcf,
                treepm_gradient=2, treepm_assignment=2, treepm_window_floor=0.0, treepm_node_size_factor=1e-6,
                multipole_order=1, octree_softening=0.02 / side) as e:
        e.set_state(pos, None, np.full(n, 1.0 / n, np.float32))
        e.accelerations()
        _, evaluated, nodes = e.walk_counts()
    assert nodes == 0
    tree = cKDTree(pos.astype(np.float64), boxsize=1.0)
    lo, hi = (tree.count_neighbors(tree, rcf / 64 * f) for f in (1 - 2e-6, 1 + 2e-6))
    assert lo <= evaluated <= hi, (lo, evaluated, hi)
